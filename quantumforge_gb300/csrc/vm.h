// vm.h — register-tile passes run from an op stream: the records shared by the
// host lowering (vmplan.cpp) and the kernels (vmpass.cuh).
//
// A CTA of 32 << W threads holds a tile of 2^K amplitudes, K = 5 + R + W:
// every thread keeps 2^R of them in registers. The thread bits (5 lane bits, W
// warp bits) and the R register bits each stand for one tile bit ("slot",
// slot s = the s-th resident qubit in ascending order); a remap through shared
// memory changes the assignment.
#pragma once

#include <cstdint>
#include <vector>

#include "qf_internal.h"

namespace qf {

constexpr int kVmMaxThreadBits = 8;  // 5 lane bits + up to 3 warp bits
constexpr int kVmMaxSlots = 12;      // tile bits
constexpr int kVmRecWords = 12;      // 48-byte op records
// Records of one launch. They travel as a kernel parameter (constant bank:
// uniform operands, no upload), which costs 0.5 us of launch time at 11 KB and
// 1.5 us at 32 KB; a pass with more records is cut into several launches.
constexpr int kVmCapacity = 240;

// Op kinds; the register bit is added to the kinds that have one.
enum VmKind : uint32_t {
    VM_FRE = 0,      // + bit: x' = x + r0 y, y' = y + r1 x, r real
    VM_FIM = 4,      // + bit: the same with r imaginary
    VM_DIAG = 8,     // + bit: registers with the bit times f
    VM_DIAGP = 12,   // registers of a 16-bit pattern times f
    VM_TPH = 13,     // thread phase times f
    VM_FLUSHP = 14,  // thread phase into the registers
    VM_REMAP = 15,   // through shared memory into a new layout
    VM_GEN = 16,     // + bit: dense complex 2x2 in the records that follow
    VM_CX = 20,      // + 4 * control bit + target bit: exchange where the control register bit is set
    VM_NEG = 36,     // + pair index (vm_pair): negate where both register bits are set
    VM_TPH2 = 42,    // thread phase times f0 or f1
    VM_SGN = 43,     // sign mask ^= A & B, each a register pattern xor a condition
    VM_FLUSHS = 44,  // signs into the registers
    VM_SCALE = 45,   // registers times a real number
    VM_OVX = 46,     // + bit: Im<lambda|X psi> into a slot
    VM_OVY = 50,     // + bit
    VM_OVZ = 54,     // the products shared by the Z overlaps that follow
    VM_OVZS = 55     // one Z overlap: register bit sum (or total), into a slot
};
constexpr int vm_pair(int a, int b) { return a + b * (b - 1) / 2; }  // a < b < 4

// One record: w0 = kind | length << 8 | flags << 16, w1 = aux, w2 = tm | tm of a
// second condition << 16, w4..7 payload, w8/w9 = qm, w10/w11 the second
// condition's. A condition is the parity of (tid & tm) and of the tile's outside
// bits & qm.
struct alignas(16) VmRec {
    uint32_t w[kVmRecWords] = {0};
};
static_assert(sizeof(VmRec) == 48, "VmRec layout");

struct VmTileOff {
    uint64_t qm, col;
};

struct VmHead {
    uint64_t nonlocal_mask;  // qubits outside the tile
    uint64_t n_tiles;
    uint64_t dim;            // 2^n: addresses at or above it (padding bits) hold no amplitude
    uint64_t sconst;         // store address: constant part
    uint64_t lcol[kVmMaxThreadBits], lreg[4];  // load address bits of the thread and register bits
    uint64_t scol[kVmMaxThreadBits], sreg[4];  // the same at the store
    VmTileOff soff[kVmMaxSlots];               // store address: parts that depend on the tile's outside bits
    uint32_t n_soff;
    uint32_t n_recs;
    uint32_t slot_base, n_ovl;  // overlap slots of this launch
    uint32_t accumulate;         // add to the partial sums of an earlier launch of the pass
};

struct VmArgs {
    VmHead h;
    VmRec recs[kVmCapacity];
};

// Takes each launch as soon as it is lowered: the GPU runs the first passes of a
// plan while the host lowers the next ones.
struct VmSink {
    virtual ~VmSink() = default;
    virtual int launch(const VmHead &h, const VmRec *recs) = 0;
};

// ---- noisy shots: one CTA per trajectory (vmtraj.cu) -------------------------
// A circuit with channels and measurements as runs of random decisions with
// unitary record streams between them.
enum TrajKind : uint8_t { TR_AD, TR_PD, TR_TH, TR_DEP, TR_MEAS };
struct TrajStep {
    uint8_t kind;
    uint8_t pos;    // the qubit in the run's layout: register bit, or 4 + thread bit
    uint8_t sd;     // state-dependent steps (all but TR_DEP): their number in the run
    uint8_t later;  // a state-dependent step on the same qubit follows in the run
    uint32_t cbit;
    double p, gu;                // probability, gamma or gamma_down; gamma_up
    double sp, s1p, su, s1u;     // square roots of p, 1 - p, gu, 1 - gu
};
struct TrajRun {
    uint32_t rec_begin, n_recs;    // the unitary part before the decisions
    uint32_t step_begin, n_steps;
    uint32_t n_sd;                 // at most one per qubit, the first R of them on register bits 0, 1, ...
    uint32_t terminal;             // measurements of distinct qubits with nothing after them
};
struct TrajProgram {
    int R = 4, W = 3;
    uint32_t n = 0;
    uint64_t lcol[kVmMaxThreadBits] = {0}, lreg[4] = {0};  // state address bits of the layout at the start
    std::vector<VmRec> recs;
    std::vector<TrajRun> runs;
    std::vector<TrajStep> steps;
};
constexpr uint32_t kTrajMaxQubits = 12;
// *ok = false: a circuit the program form does not cover (feed-forward, invalid
// operations).
int vm_lower_trajectories(uint32_t n, const qf_op *ops, uint64_t n_ops, TrajProgram &out, bool *ok);
int run_trajectories_vm(qf_sv *init, const TrajProgram &prog, uint64_t shots, const uint64_t *starts, double tie_eps,
                        uint64_t *outcomes, uint64_t *n_ties);

// Register and warp bits of a tile of k bits.
void vm_shape(int k, int dtype, bool dual, int *R, int *W);
// The widest tile the passes take, and the one they use when the caller names none.
int vm_widest(int dtype, bool dual);
int vm_default_tile(uint32_t n, int dtype, bool dual);
// Lower a forward plan (dual: a backward plan with overlaps) to op streams on
// tiles of R register and W warp bits.
int vm_lower(const Plan &plan, int dtype, int R, int W, VmSink &sink);
int run_plan_vm(qf_sv *sv, const Plan &plan);
// Backward passes; complex128 only.
int run_plan_vm_dual(qf_sv *psi, qf_sv *lam, const Plan &plan, double *d_slot_sums);

}  // namespace qf
