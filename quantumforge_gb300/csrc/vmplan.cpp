// vmplan.cpp — host lowering of tile-pass plans to the op streams of the
// register-tile kernels (vm.h, vmpass.cuh). No device code.
//
// A pass's gates are first scheduled: gates commute unless they share a qubit on
// which one of them is not diagonal, a dense gate runs while its qubit is in
// a register position, and when nothing can run the tile is remapped to the
// layout that lets the most gates run. The schedule depends only on the pass's
// structure and is cached under it.
//
// Emission then walks the schedule and keeps everything that needs no
// arithmetic on the amplitudes symbolic:
//  * each tile bit is an affine function of the thread's bits, the tile's
//    outside bits and at most one register bit, so X gates, SWAPs and CNOTs
//    whose control is not in a register are index bookkeeping;
//  * CZs and Z gates are a sign frame (a quadratic form of the qubits' bits); a
//    dense gate on a qubit takes its linear part there as a sign of its
//    coefficients, and the form stays;
//  * diagonal gates wait as phase terms f^parity(mask) until a dense gate acts
//    on one of their qubits. Terms on bits that a thread's registers share cost
//    one complex multiply per thread; they are folded into the registers together
//    before a remap, once enough of them wait;
//  * scalar factors pulled out of gates multiply into one number.
// Frames, terms and the scalar travel from pass to pass and are applied by the
// last launch of the plan.
//
// Every dense gate becomes x' = x + r0 y, y' = y + r1 x with r real or imaginary:
// a real or RX-type unitary has that form up to a factor, an X and a Z
// (factor_unitary_2x2), any other unitary is diag * real rotation * diag. Two FP
// operations per amplitude, which is what bounds complex128 passes.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <unordered_map>

#include "vm.h"

namespace qf {

using cd = std::complex<double>;

// complex128: at least four warps as soon as the tile allows (one warp reaches
// 0.5 FP64 lanes per clock, an SM 1.7), then registers; complex64: as many
// registers as there are, which leaves the fewest remaps.
void vm_shape(int k, int dtype, bool dual, int *R, int *W) {
    const int K = std::max(k, 6);
    const int most = dual && dtype == QF_C128 ? 3 : 4;
    *R = dtype == QF_C128 ? std::min(std::max(K - 7, 1), most) : std::min(K - 5, most);
    *W = K - 5 - *R;
}

int vm_widest(int dtype, bool dual) { return dual && dtype == QF_C128 ? 11 : 12; }

// complex128 is priced by its FP64 work, so small tiles win while they are what
// spreads it over the SMs (8 bits: 14 qubits in 199 us against 279 with 10 and
// 732 with 12, one depth-20 circuit; 9 bits: 18 qubits in 475 against 881 with
// 12), until the extra passes cost more (22 qubits: 6.18 ms with 12, 6.37 with
// 9). complex64 is priced by records and launches: wide tiles, 11 bits with half
// the threads a little ahead of 12 (21 qubits: 454 against 481 us).
int vm_default_tile(uint32_t n, int dtype, bool dual) {
    if (dtype == QF_C64) return n <= 12 ? (int)n : 11;
    if (n <= 8) return (int)n;
    if (n <= 14) return 8;
    if (dual) return n <= 17 ? 9 : n == 18 ? 10 : 11;
    return n <= 20 ? 9 : n == 21 ? 10 : 12;
}

namespace {

constexpr int kNone = -1;

struct Layout {
    int8_t tslot[kVmMaxThreadBits];
    int8_t rslot[4];
};

struct Step {
    int gate;    // index into the pass's gates, or
    int layout;  // remap to this layout
};

struct Sched {
    std::vector<Step> steps;
    std::vector<Layout> layouts;  // [0]: at load
};

enum GClass : uint8_t { G_DENSE, G_DIAG, G_ANTI, G_CNOT, G_CZ, G_SWAP, G_OVZ, G_OVXY };

// Up to the rounding of a product of gates. Kraus operators carry a flag: those of
// a weak channel are as close to unitary as that.
bool unit(cd f) { return std::abs(std::abs(f) - 1.0) < 1e-9; }
bool anti_diagonal(const BGate &g) {  // a unitary one (not the jump operator of a damping channel)
    const double *m = g.m;
    return !g.kraus && m[0] == 0 && m[1] == 0 && m[6] == 0 && m[7] == 0 && unit(cd(m[2], m[3])) && unit(cd(m[4], m[5]));
}

GClass class_of(const BGate &g) {
    switch (g.kind) {
    case BK_MAT1: return g.diag ? G_DIAG : anti_diagonal(g) ? G_ANTI : G_DENSE;
    case BK_CNOT: return G_CNOT;
    case BK_CZ: return G_CZ;
    case BK_SWAP: return G_SWAP;
    default: return g.axis == QF_PAULI_Z ? G_OVZ : G_OVXY;
    }
}

// Swizzled shared-memory index of one tile bit (XOR-linear): complex64
// half-warps want lane bits 0..3 to reach all four bits of an 8-byte index,
// complex128 quarter-warps lane bits 0..2 the three bits of a 16-byte index. The
// folded vectors leave a basis among any eight slots of twelve.
uint32_t phys_bit(int s, int dtype) {
    static const uint32_t v4[8] = {3, 5, 6, 9, 10, 12, 7, 11}, v3[9] = {3, 5, 6, 7, 1, 2, 4, 3, 5};
    if (dtype == QF_C64) return (1u << s) ^ (s >= 4 ? v4[s - 4] : 0u);
    return (1u << s) ^ (s >= 3 ? v3[s - 3] : 0u);
}
uint32_t bank_bits(int s, int dtype) { return phys_bit(s, dtype) & (dtype == QF_C64 ? 15u : 7u); }

// Lanes hold the lowest `low` tile bits at load and store: 128-byte runs.
int low_bits(int dtype) { return dtype == QF_C64 ? 4 : 3; }

struct PassSlots {
    int K, R, NT;           // tile bits (with padding), register bits, thread bits
    int k;                  // tile bits that are qubits
    uint32_t slot_q[kVmMaxSlots];
    int slot_of[64];
    PassSlots(const Pass &p, uint32_t n, int R_, int W) : K(5 + R_ + W), R(R_), NT(5 + W), k(0) {
        for (int q = 0; q < 64; ++q) slot_of[q] = kNone;
        for (uint32_t q = 0; q < n; ++q)
            if ((p.resident >> q) & 1ULL) {
                slot_of[q] = k;
                slot_q[k++] = q;
            }
    }
    uint64_t address_bit(int s) const { return s < k ? 1ULL << slot_q[s] : 1ULL << (48 + s); }  // padding: above any state
};

// A layout with `regs` (at most R slots) in the register bits, the others filled
// from the highest free slots; lanes with independent bank bits first (remap) or
// the lowest slots in order (load, store).
Layout make_layout(const PassSlots &ps, uint32_t regs, bool natural, int dtype) {
    Layout L;
    int nr = 0;
    uint32_t used = 0;
    for (int s = 0; s < ps.K; ++s)
        if ((regs >> s) & 1u) {
            L.rslot[nr++] = (int8_t)s;
            used |= 1u << s;
        }
    for (int s = ps.k - 1; s >= 0 && nr < ps.R; --s)
        if (!((used >> s) & 1u)) {
            L.rslot[nr++] = (int8_t)s;
            used |= 1u << s;
        }
    for (int s = ps.K - 1; s >= 0 && nr < ps.R; --s)
        if (!((used >> s) & 1u)) {
            L.rslot[nr++] = (int8_t)s;
            used |= 1u << s;
        }
    int nt = 0;
    if (!natural) {
        const int want = dtype == QF_C64 ? 4 : 3;
        uint32_t basis[4];
        int nb = 0;
        for (int s = 0; s < ps.K && nt < want; ++s) {
            if ((used >> s) & 1u) continue;
            uint32_t v = bank_bits(s, dtype);
            for (int i = 0; i < nb; ++i) v = std::min(v, v ^ basis[i]);
            if (!v) continue;
            basis[nb++] = v;
            L.tslot[nt++] = (int8_t)s;
            used |= 1u << s;
        }
    }
    for (int s = 0; s < ps.K; ++s)
        if (!((used >> s) & 1u)) {
            L.tslot[nt++] = (int8_t)s;
            used |= 1u << s;
        }
    for (; nt < kVmMaxThreadBits; ++nt) L.tslot[nt] = kNone;
    for (; nr < 4; ++nr) L.rslot[nr] = kNone;
    return L;
}

// ---- scheduling ---------------------------------------------------------------
struct Scheduler {
    const std::vector<BGate> &G;
    const PassSlots &ps;
    int dtype;
    std::vector<GClass> cls;
    std::vector<int> s0, s1;                // tile bits of the gate's qubits
    std::vector<std::vector<int>> preds;
    std::vector<char> done;
    std::vector<int> todo;                  // not yet run, in order

    Scheduler(const std::vector<BGate> &gates, const PassSlots &p, int dt) : G(gates), ps(p), dtype(dt) {
        const size_t n = G.size();
        cls.resize(n);
        s0.resize(n);
        s1.resize(n);
        preds.resize(n);
        done.assign(n, 0);
        int last[64];                     // last gate not diagonal on the qubit
        std::vector<int> since[64];       // gates diagonal on it since
        for (int q = 0; q < 64; ++q) last[q] = kNone;
        for (size_t j = 0; j < n; ++j) {
            const BGate &g = G[j];
            cls[j] = class_of(g);
            const bool two = cls[j] == G_CNOT || cls[j] == G_CZ || cls[j] == G_SWAP;
            s0[j] = ps.slot_of[g.q0];
            s1[j] = two ? ps.slot_of[g.q1] : kNone;
            for (int a = 0; a < (two ? 2 : 1); ++a) {
                const uint32_t q = a ? g.q1 : g.q0;
                const bool diag = cls[j] == G_DIAG || cls[j] == G_CZ || cls[j] == G_OVZ || (cls[j] == G_CNOT && a == 0);
                if (diag) {
                    if (last[q] != kNone) preds[j].push_back(last[q]);
                    since[q].push_back((int)j);
                } else {
                    if (since[q].empty()) {
                        if (last[q] != kNone) preds[j].push_back(last[q]);
                    } else {
                        preds[j].insert(preds[j].end(), since[q].begin(), since[q].end());
                    }
                    since[q].clear();
                    last[q] = (int)j;
                }
            }
            todo.push_back((int)j);
        }
    }
    bool ready(int j, const std::vector<char> &d) const {
        for (int i : preds[j])
            if (!d[i]) return false;
        return true;
    }
    static bool in(uint32_t regs, int s) { return s >= 0 && ((regs >> s) & 1u); }
    bool runnable(int j, uint32_t regs) const {
        switch (cls[j]) {
        case G_DENSE:
        case G_OVXY: return in(regs, s0[j]);
        case G_CNOT: return in(regs, s1[j]) || !in(regs, s0[j]);
        default: return true;
        }
    }
    // SWAPs exchange register membership
    static uint32_t after(uint32_t regs, GClass c, int a, int b) {
        if (c == G_SWAP && in(regs, a) != in(regs, b)) regs ^= (1u << a) | (1u << b);
        return regs;
    }
    // gates (weighted: those that need registers first) run under `regs`
    int simulate(uint32_t regs) const {
        std::vector<char> d = done;
        int dense = 0, all = 0;
        for (int j : todo) {
            if (!ready(j, d) || !runnable(j, regs)) continue;
            d[j] = 1;
            ++all;
            dense += cls[j] == G_DENSE || cls[j] == G_OVXY || cls[j] == G_CNOT;
            regs = after(regs, cls[j], s0[j], s1[j]);
        }
        return dense * 4096 + all;
    }
    // R tile bits from `allowed`, greedily the one that lets the most run (the
    // highest on ties: low bits suit lanes). A CNOT's control in a register holds
    // the gate up while its target is not, so every register is chosen this way.
    uint32_t choose(uint32_t allowed) const {
        uint32_t S = 0;
        for (int c = 0; c < ps.R; ++c) {
            int pick = kNone, pb = -1;
            for (int s = ps.K - 1; s >= 0; --s) {
                if (!((allowed >> s) & 1u) || in(S, s)) continue;
                const int v = simulate(S | (1u << s));
                if (v > pb) {
                    pb = v;
                    pick = s;
                }
            }
            if (pick == kNone) break;
            S |= 1u << pick;
        }
        return S;
    }
    bool run(Sched &out, const Layout *start) {
        const uint32_t low = (1u << std::min(low_bits(dtype), ps.k)) - 1u;
        const uint32_t every = (1u << ps.K) - 1u;
        // small tiles: registers must leave the lanes some bits
        const uint32_t first = ps.K - __builtin_popcount(low) >= ps.R ? every & ~low : every;
        out.layouts.push_back(start ? *start : make_layout(ps, choose(first), true, dtype));
        uint32_t regs = 0;
        auto set_regs = [&] {
            regs = 0;
            for (int r = 0; r < ps.R; ++r) regs |= 1u << out.layouts.back().rslot[r];
        };
        set_regs();
        bool fresh = true;
        while (!todo.empty()) {
            bool progress = false;
            for (bool again = true; again;) {  // SWAPs and releases can make earlier gates runnable
                again = false;
                size_t w = 0;
                for (size_t r = 0; r < todo.size(); ++r) {
                    const int j = todo[r];
                    if (cls[j] != G_OVZ && ready(j, done) && runnable(j, regs)) {
                        done[j] = 1;
                        out.steps.push_back({j, kNone});
                        regs = after(regs, cls[j], s0[j], s1[j]);
                        again = progress = true;
                    } else {
                        todo[w++] = j;
                    }
                }
                todo.resize(w);
            }
            if (todo.empty()) break;
            // Z overlaps wait until nothing else runs, then share their products
            size_t w = 0;
            bool z = false;
            for (size_t r = 0; r < todo.size(); ++r) {
                const int j = todo[r];
                if (cls[j] == G_OVZ && ready(j, done)) {
                    out.steps.push_back({j, kNone});
                    z = true;
                    done[j] = 2;  // released below: overlaps of one group see the same gates
                } else {
                    todo[w++] = j;
                }
            }
            todo.resize(w);
            for (char &d : done)
                if (d == 2) d = 1;
            if (z) {
                fresh = false;
                continue;
            }
            if (!progress && fresh && out.layouts.size() > 1) return false;  // a remap that released nothing
            out.layouts.push_back(make_layout(ps, choose(every), false, dtype));
            out.steps.push_back({kNone, (int)out.layouts.size() - 1});
            set_regs();
            fresh = true;
        }
        return true;
    }
};

struct SchedCache {
    std::mutex mu;
    std::unordered_map<std::string, std::shared_ptr<const Sched>> entries;
};
SchedCache &sched_cache() {
    static SchedCache c;
    return c;
}
constexpr size_t kSchedEntries = 4096;

// The pass's schedule; start: the layout its amplitudes already have.
std::shared_ptr<const Sched> schedule(const Pass &p, const PassSlots &ps, uint32_t n, int dtype, const Layout *start = nullptr) {
    std::string key;
    key.reserve(11 + 3 * p.gates.size());
    key.append(reinterpret_cast<const char *>(&p.resident), 8);
    key.push_back((char)n);
    key.push_back((char)(ps.R | (ps.NT << 3)));
    key.push_back((char)(dtype | (start ? 2 : 0)));
    if (start) key.append(reinterpret_cast<const char *>(start), sizeof *start);
    for (const BGate &g : p.gates) {
        const char e[3] = {(char)class_of(g), (char)g.q0, (char)g.q1};
        key.append(e, 3);
    }
    {
        std::lock_guard<std::mutex> lk(sched_cache().mu);
        auto it = sched_cache().entries.find(key);
        if (it != sched_cache().entries.end()) return it->second;
    }
    auto s = std::make_shared<Sched>();
    if (!Scheduler(p.gates, ps, dtype).run(*s, start)) return nullptr;
    std::lock_guard<std::mutex> lk(sched_cache().mu);
    if (sched_cache().entries.size() >= kSchedEntries) sched_cache().entries.clear();  // bound the host memory
    sched_cache().entries[key] = s;
    return s;
}

// ---- emission -------------------------------------------------------------------
// A tile bit (or outside qubit) as an affine function: register bit `reg` (or
// none) ^ parity(tid & T) ^ parity(outside bits & Q) ^ k.
struct Fn {
    int reg = kNone;
    uint32_t T = 0;
    uint64_t Q = 0;
    uint32_t k = 0;
    bool pure() const { return T == 0 && Q == 0; }
};

struct Term {  // the phase f^parity(x & mask), |f| = 1
    uint64_t mask;
    cd f;
};

// The product of the factors pulled out of gates: hundreds of them, so both
// parts are kept as unevaluated pairs of doubles and the product adds no
// rounding of its own to the state.
struct Scalar {
    double r[2] = {1.0, 0.0}, i[2] = {0.0, 0.0};
    static void fma2(double acc[2], const double x[2], double y) {  // acc += x y
        const double p = x[0] * y, e = std::fma(x[0], y, -p) + x[1] * y;
        const double s = acc[0] + p, b = s - acc[0];
        const double t = (acc[0] - (s - b)) + (p - b) + acc[1] + e;
        acc[0] = s + t;
        acc[1] = t - (acc[0] - s);
    }
    void operator*=(cd f) {
        double a[2] = {0.0, 0.0}, b[2] = {0.0, 0.0};
        fma2(a, r, f.real());
        fma2(a, i, -f.imag());
        fma2(b, r, f.imag());
        fma2(b, i, f.real());
        std::memcpy(r, a, sizeof a);
        std::memcpy(i, b, sizeof b);
    }
    void negate() {
        for (double *x : {r, i}) x[0] = -x[0], x[1] = -x[1];
    }
    cd value() const { return {r[0], i[0]}; }
    bool is_one() const { return r[0] == 1.0 && r[1] == 0.0 && i[0] == 0.0 && i[1] == 0.0; }
    double abs() const { return std::abs(value()); }
};

struct Emitter {
    const Plan &plan;
    int dtype;
    VmSink &sink;
    std::vector<VmRec> recs;  // of the open launch
    VmHead head;
    // carried from pass to pass
    std::vector<Term> terms;
    uint64_t zmask = 0;          // sign frame: (-1)^(x & zmask)
    uint64_t adj[64] = {0};      // and (-1)^(x_a x_b) for every b in adj[a]
    Scalar scale;
    // of the pass
    const Pass *pass = nullptr;
    const PassSlots *ps = nullptr;
    Fn fn[kVmMaxSlots];
    bool tph = false;         // a thread phase waits
    std::vector<int> later;   // per qubit: dense gates of this pass still to come

    Emitter(const Plan &p, int dt, VmSink &s) : plan(p), dtype(dt), sink(s) { recs.reserve(kVmCapacity); }

    Fn fn_of(uint32_t q) const {
        const int s = ps->slot_of[q];
        if (s >= 0) return fn[s];
        Fn f;
        f.Q = 1ULL << q;
        return f;
    }
    VmRec &rec(uint32_t kind, const Fn *c = nullptr, uint32_t len = 1) {
        recs.emplace_back();
        VmRec &r = recs.back();
        r.w[0] = kind | (len << 8);
        if (c) {
            r.w[2] = c->T;
            r.w[8] = (uint32_t)c->Q;
            r.w[9] = (uint32_t)(c->Q >> 32);
        }
        return r;
    }
    static void second(VmRec &r, const Fn &c) {
        r.w[2] |= c.T << 16;
        r.w[10] = (uint32_t)c.Q;
        r.w[11] = (uint32_t)(c.Q >> 32);
    }
    void put(uint32_t *w, int i, double v) const {
        if (dtype == QF_C64) {
            const float f = (float)v;
            std::memcpy(w + i, &f, 4);
        } else {
            std::memcpy(w + 2 * i, &v, 8);
        }
    }

    uint32_t regs_of(uint64_t mask, Fn *rest) const {  // register part of a parity, the remainder in *rest
        uint32_t rm = 0;
        Fn f;
        for (uint64_t m = mask; m; m &= m - 1) {
            const Fn g = fn_of((uint32_t)__builtin_ctzll(m));
            if (g.reg != kNone) rm ^= 1u << g.reg;
            f.T ^= g.T;
            f.Q ^= g.Q;
            f.k ^= g.k;
        }
        *rest = f;
        return rm;
    }
    static uint32_t pattern(uint32_t rm) {  // bit i: parity(i & rm)
        uint32_t p = 0;
        for (uint32_t i = 0; i < 16; ++i) p |= (uint32_t)(__builtin_popcount(i & rm) & 1) << i;
        return p;
    }

    void add_term(uint64_t mask, cd f) {
        if (f == cd(1.0, 0.0)) return;
        for (size_t i = 0; i < terms.size(); ++i)
            if (terms[i].mask == mask) {
                terms[i].f *= f;
                if (terms[i].f == cd(1.0, 0.0)) terms.erase(terms.begin() + (long)i);
                return;
            }
        terms.push_back({mask, f});
    }
    // one term onto the amplitudes
    void apply_term(const Term &t) {
        Fn r;
        const uint32_t rm = regs_of(t.mask, &r);
        if (!rm) {
            VmRec &w = rec(VM_TPH, &r);
            w.w[0] |= r.k << 16;
            put(w.w + 4, 0, t.f.real());
            put(w.w + 4, 1, t.f.imag());
            tph = true;
            return;
        }
        cd f = t.f;
        if (r.k) {  // f^(1 ^ b) = f (1/f)^b
            scale *= f;
            f = std::conj(f);
        }
        const bool one = (rm & (rm - 1)) == 0;
        VmRec &w = rec(one ? VM_DIAG + (uint32_t)__builtin_ctz(rm) : (uint32_t)VM_DIAGP, &r);
        w.w[0] |= r.pure() ? 0u : 1u << 16;
        w.w[1] = pattern(rm);
        put(w.w + 4, 0, f.real());
        put(w.w + 4, 1, f.imag());
        tph = tph || !r.pure();
    }
    void apply_terms_on(uint64_t qmask) {
        for (size_t i = 0; i < terms.size();)
            if (terms[i].mask & qmask) {
                apply_term(terms[i]);
                terms.erase(terms.begin() + (long)i);
            } else {
                ++i;
            }
    }
    void flush_phase() {
        if (!tph) return;
        if (scale.abs() < 0x1p-16) {  // the scalar rides along
            emit_scalar_phase();
        }
        rec(VM_FLUSHP);
        tph = false;
    }
    void emit_scalar_phase() {
        VmRec &w = rec(VM_TPH);
        w.w[0] |= 1u << 16;  // every thread
        put(w.w + 4, 0, scale.value().real());
        put(w.w + 4, 1, scale.value().imag());
        scale = Scalar();
        tph = true;
    }
    // the sign (-1)^(parity(x & ma) parity(x & mb)), mb = 0 for the first factor alone
    void emit_sign(uint64_t ma, uint64_t mb) {
        Fn a, b;
        const uint32_t ra = regs_of(ma, &a), rb = mb ? regs_of(mb, &b) : 0;
        VmRec &w = rec(VM_SGN, &a);
        const uint32_t pa = pattern(ra) ^ (a.k ? 0xFFFFu : 0u);
        const uint32_t pb = mb ? pattern(rb) ^ (b.k ? 0xFFFFu : 0u) : 0xFFFFu;
        w.w[1] = (pa << 16) | pb;
        if (mb) second(w, b);
    }

    // Thread-level terms are folded into the registers together: one complex
    // multiply per amplitude against half a one for each term applied alone in a
    // register (complex64 also pays each record's dispatch).
    void before_remap() {
        int wanted = 0;
        for (const Term &t : terms) {
            Fn r;
            if (regs_of(t.mask, &r)) continue;
            bool need = false;
            for (uint64_t m = t.mask; m; m &= m - 1) need = need || later[__builtin_ctzll(m)] > 0;
            wanted += need;
        }
        if (tph || wanted >= (dtype == QF_C64 ? 2 : 3)) {
            for (size_t i = 0; i < terms.size();) {
                Fn r;
                if (regs_of(terms[i].mask, &r)) {
                    ++i;
                    continue;
                }
                apply_term(terms[i]);
                terms.erase(terms.begin() + (long)i);
            }
        }
        flush_phase();
    }
    void emit_remap(const Layout &L) {
        before_remap();
        uint32_t wcol[kVmMaxThreadBits] = {0}, rcol[kVmMaxThreadBits] = {0}, wreg[4] = {0}, rreg[4] = {0}, wconst = 0;
        VmTileOff offs[kVmMaxSlots];
        size_t n_off = 0;
        for (int s = 0; s < ps->K; ++s) {
            const uint32_t pb = phys_bit(s, dtype);
            for (int i = 0; i < ps->NT; ++i)
                if ((fn[s].T >> i) & 1u) wcol[i] ^= pb;
            if (fn[s].reg != kNone) wreg[fn[s].reg] ^= pb;
            if (fn[s].k) wconst ^= pb;
            if (fn[s].Q) offs[n_off++] = {fn[s].Q, pb};
        }
        for (int i = 0; i < ps->NT; ++i) rcol[i] = phys_bit(L.tslot[i], dtype);
        for (int r = 0; r < ps->R; ++r) rreg[r] = phys_bit(L.rslot[r], dtype);
        VmRec &w = rec(VM_REMAP, nullptr, (uint32_t)(2 + (n_off + 1) / 2));
        w.w[1] = (uint32_t)n_off;
        w.w[2] = wreg[0] | (wreg[1] << 16);
        w.w[3] = wreg[2] | (wreg[3] << 16);
        w.w[4] = rreg[0] | (rreg[1] << 16);
        w.w[5] = rreg[2] | (rreg[3] << 16);
        w.w[6] = wconst;
        VmRec &c = rec(0);
        for (int i = 0; i < 4; ++i) {
            c.w[i] = wcol[2 * i] | (wcol[2 * i + 1] << 16);
            c.w[4 + i] = rcol[2 * i] | (rcol[2 * i + 1] << 16);
        }
        for (size_t k = 0; k < n_off; k += 2) {
            VmRec &f = rec(0);
            for (size_t e = 0; e < 2 && k + e < n_off; ++e) {
                f.w[3 * e] = (uint32_t)offs[k + e].qm;
                f.w[3 * e + 1] = (uint32_t)(offs[k + e].qm >> 32);
                f.w[3 * e + 2] = (uint32_t)offs[k + e].col;
            }
        }
        set_layout(L);
    }
    void set_layout(const Layout &L) {
        for (Fn &f : fn) f = Fn();
        for (int i = 0; i < ps->NT; ++i) fn[(int)L.tslot[i]].T = 1u << i;
        for (int r = 0; r < ps->R; ++r) fn[(int)L.rslot[r]].reg = r;
    }

    // The sign frame around an operation on register qubit q: the parity of q's
    // neighbours as the returned function; neighbours that sit in registers are
    // settled in the amplitudes (the pair leaves the frame) where both bits are
    // plain, otherwise negations before and after the operation (`around`) stand
    // for them.
    Fn neighbours(uint32_t q, std::vector<uint32_t> &around) {
        const Fn fq = fn_of(q);
        Fn L;
        for (uint64_t m = adj[q]; m; m &= m - 1) {
            const uint32_t b = (uint32_t)__builtin_ctzll(m);
            const Fn fb = fn_of(b);
            if (fb.reg != kNone) {
                const uint32_t kind = VM_NEG + (uint32_t)vm_pair(std::min(fq.reg, fb.reg), std::max(fq.reg, fb.reg));
                if (fq.pure() && fb.pure()) {  // x_q x_b = i_q i_b ^ k_b x_q ^ k_q x_b ^ k_q k_b
                    rec(kind);
                    toggle(q, b);
                    if (fb.k) zmask ^= 1ULL << q;
                    if (fq.k) zmask ^= 1ULL << b;
                    if (fq.k && fb.k) scale.negate();
                    continue;
                }
                around.push_back(kind);
            }
            L.T ^= fb.T;
            L.Q ^= fb.Q;
            L.k ^= fb.k;
        }
        for (uint32_t k : around) rec(k);
        return L;
    }
    void toggle(uint32_t a, uint32_t b) {
        adj[a] ^= 1ULL << b;
        adj[b] ^= 1ULL << a;
    }

    // a dense 2x2 on a register qubit as plain complex multiplies
    void emit_general(uint32_t q, const cd m_[4], const Fn &L) {
        const Fn f = fn_of(q);
        cd m[4] = {m_[0], m_[1], m_[2], m_[3]};
        if (f.k) {
            std::swap(m[0], m[3]);
            std::swap(m[1], m[2]);
        }
        if (L.k) {
            m[1] = -m[1];
            m[2] = -m[2];
        }
        second(rec(VM_GEN + (uint32_t)f.reg, &f, dtype == QF_C64 ? 2 : 3), L);
        VmRec *a = &rec(0);
        for (int e = 0; e < 4; ++e) {
            if (e == 2 && dtype == QF_C128) a = &rec(0);
            const int at = dtype == QF_C128 ? 2 * (e & 1) : 2 * e;
            put(a->w, at, m[e].real());
            put(a->w, at + 1, m[e].imag());
        }
    }
    // x' = x + r0 y, y' = y + r1 x (both real or both imaginary)
    void emit_factored(uint32_t q, cd r0, cd r1, bool imag, const Fn &L) {
        if (r0 == cd(0.0, 0.0) && r1 == cd(0.0, 0.0)) return;
        const Fn f = fn_of(q);
        if (f.k) std::swap(r0, r1);
        const double s = L.k ? -1.0 : 1.0;
        VmRec &w = rec((imag ? VM_FIM : VM_FRE) + (uint32_t)f.reg, &f);
        w.w[0] |= ((f.pure() ? 0u : 1u) | (L.pure() ? 0u : 2u)) << 16;
        put(w.w + 4, 0, s * (imag ? r0.imag() : r0.real()));
        put(w.w + 4, 1, s * (imag ? r1.imag() : r1.real()));
        second(w, L);
    }
    static void flip_column(cd m[4]) {
        m[1] = -m[1];
        m[3] = -m[3];
    }
    void emit_dense(uint32_t q, const double md[8], bool kraus) {
        cd m[4] = {{md[0], md[1]}, {md[2], md[3]}, {md[4], md[5]}, {md[6], md[7]}};
        double mm[8];
        auto factor = [&] {
            for (int e = 0; e < 4; ++e) {
                mm[2 * e] = m[e].real();
                mm[2 * e + 1] = m[e].imag();
            }
            return factor_unitary_2x2(mm);
        };
        Factored f = kraus ? Factored() : factor();
        cd after(1.0, 0.0);
        if (!f.ok && !kraus) {
            const double n0 = std::norm(m[0]) + std::norm(m[2]), n1 = std::norm(m[1]) + std::norm(m[3]);
            const cd dot = std::conj(m[0]) * m[1] + std::conj(m[2]) * m[3];
            const bool unitary = std::abs(n0 - 1.0) < 1e-9 && std::abs(n1 - 1.0) < 1e-9 && std::abs(dot) < 1e-9;
            if (unitary && m[0] != 0.0 && m[1] != 0.0 && m[2] != 0.0) {  // u diag(1, a) rotation diag(1, b)
                const cd u = m[0] / std::abs(m[0]);
                const cd a = m[2] / std::abs(m[2]) / u, b = -m[1] / std::abs(m[1]) / u;
                const double c = std::sqrt(0.5 * (std::norm(m[0]) + std::norm(m[3])));
                const double s = std::sqrt(0.5 * (std::norm(m[1]) + std::norm(m[2])));
                scale *= u;
                add_term(1ULL << q, b);
                after = a;
                m[0] = m[3] = c;
                m[1] = -s;
                m[2] = s;
                f = factor();
            }
        }
        apply_terms_on(1ULL << q);
        std::vector<uint32_t> around;
        const Fn L = neighbours(q, around);
        if ((zmask >> q) & 1ULL) {  // the Z frame goes into the matrix
            zmask ^= 1ULL << q;
            flip_column(m);
            if (f.ok) f = factor();
        }
        if (!f.ok) {
            emit_general(q, m, L);
        } else {  // U = g (sigma) F, or g (sigma) X F, with F: x' = x + r0 y, y' = y + r1 x
            scale *= f.g;
            const double sg = f.neg ? -1.0 : 1.0;
            if (f.pivot == 0) {
                emit_factored(q, f.r0, sg * f.r1, f.imag_r, L);
            } else {
                emit_factored(q, sg * f.r1, f.r0, f.imag_r, L);
                fn[ps->slot_of[q]].k ^= 1u;
                zmask ^= adj[q];  // X through the frame
            }
            if (f.neg) zmask ^= 1ULL << q;
        }
        for (uint32_t k : around) rec(k);
        if (after != cd(1.0, 0.0)) add_term(1ULL << q, after);
    }
    // [[0, a], [b, 0]]: phases, then X
    void emit_anti(uint32_t q, const double m[8]) {
        const cd a(m[2], m[3]), b(m[4], m[5]);
        // out0 = a y, out1 = b x: diag(b, a) first, then the exchange
        scale *= b;
        add_term(1ULL << q, a / b);
        for (size_t i = 0; i < terms.size(); ++i)
            if ((terms[i].mask >> q) & 1ULL) {  // f^(1 ^ x) = f conj(f)^x
                scale *= terms[i].f;
                terms[i].f = std::conj(terms[i].f);
            }
        if ((zmask >> q) & 1ULL) scale.negate();
        zmask ^= adj[q];
        fn[ps->slot_of[q]].k ^= 1u;
    }
    void emit_diag(uint32_t q, const double m[8], bool kraus) {
        const cd a(m[0], m[1]), b(m[6], m[7]);
        if (!kraus && unit(a) && unit(b)) {
            scale *= a;
            const cd f = b / a;
            if (f == cd(-1.0, 0.0)) zmask ^= 1ULL << q;
            else add_term(1ULL << q, f);
            return;
        }
        // a Kraus operator: at once
        const Fn f = fn_of(q);
        if (f.reg != kNone) {
            const cd full[4] = {a, 0.0, 0.0, b};
            emit_general(q, full, Fn());
            return;
        }
        VmRec &w = rec(VM_TPH2, &f, 2);
        w.w[0] |= f.k << 16;
        VmRec &p = rec(0);
        put(p.w, 0, a.real());
        put(p.w, 1, a.imag());
        put(p.w, 2, b.real());
        put(p.w, 3, b.imag());
        tph = true;
    }
    void emit_cnot(uint32_t c, uint32_t t) {
        const Fn fc = fn_of(c);
        const int st = ps->slot_of[t];
        if (fc.reg != kNone) {  // both in registers (the schedule's rule)
            rec(VM_CX + 4u * (uint32_t)fc.reg + (uint32_t)fn[st].reg);
        }
        fn[st].T ^= fc.T;
        fn[st].Q ^= fc.Q;
        fn[st].k ^= fc.k;
        // the old value of t is t ^ c now
        for (Term &x : terms)
            if ((x.mask >> t) & 1ULL) x.mask ^= 1ULL << c;
        if ((zmask >> t) & 1ULL) zmask ^= 1ULL << c;
        const uint64_t nt = adj[t];
        if ((nt >> c) & 1ULL) zmask ^= 1ULL << c;
        for (uint64_t m = nt & ~(1ULL << c); m; m &= m - 1) toggle(c, (uint32_t)__builtin_ctzll(m));
        merge_terms();
    }
    void merge_terms() {  // masks may have become equal or empty
        for (size_t i = 0; i < terms.size(); ++i)
            for (size_t j = terms.size(); j-- > i + 1;)
                if (terms[j].mask == terms[i].mask) {
                    terms[i].f *= terms[j].f;
                    terms.erase(terms.begin() + (long)j);
                }
    }
    void emit_swap(uint32_t a, uint32_t b) {
        std::swap(fn[ps->slot_of[a]], fn[ps->slot_of[b]]);
        auto sw = [&](uint64_t m) {
            const uint64_t x = (m >> a) & 1ULL, y = (m >> b) & 1ULL;
            if (x != y) m ^= (1ULL << a) | (1ULL << b);
            return m;
        };
        for (Term &t : terms) t.mask = sw(t.mask);
        zmask = sw(zmask);
        std::swap(adj[a], adj[b]);
        for (uint64_t &m : adj) m = sw(m);
    }
    double overlap_factor() const { return std::norm(scale.value()); }
    void emit_overlap_xy(const BGate &g) {
        apply_terms_on(1ULL << g.q0);
        std::vector<uint32_t> around;
        const Fn L = neighbours(g.q0, around);
        const Fn f = fn_of(g.q0);
        double v = overlap_factor();
        if (L.k) v = -v;
        if ((zmask >> g.q0) & 1ULL) v = -v;
        if (g.axis == QF_PAULI_Y && f.k) v = -v;
        VmRec &w = rec((g.axis == QF_PAULI_Y ? VM_OVY : VM_OVX) + (uint32_t)f.reg, &f);
        w.w[1] = (uint32_t)(g.op_index - pass->a.slot_base);
        put(w.w + 4, 0, v);
        second(w, L);
        for (uint32_t k : around) rec(k);
    }
    void emit_overlap_z(const BGate &g, bool first) {
        if (first) rec(VM_OVZ);
        const Fn f = fn_of(g.q0);
        double v = overlap_factor();
        if (f.k) v = -v;
        VmRec &w = rec(VM_OVZS, &f);
        w.w[1] = (uint32_t)(g.op_index - pass->a.slot_base) | ((uint32_t)(f.reg + 1) << 16);
        put(w.w + 4, 0, v);
    }

    static constexpr int kMaxTerms = 32;
    // ---- launches ----
    void open(const Layout &L, bool again) {
        std::memset(&head, 0, sizeof head);
        head.nonlocal_mask = pass->a.nonlocal_mask;
        head.n_tiles = pass->a.n_tiles;
        head.dim = 1ULL << plan.n;
        head.slot_base = pass->a.slot_base;
        head.n_ovl = pass->a.n_slots;
        head.accumulate = again;
        for (int i = 0; i < ps->NT; ++i) head.lcol[i] = ps->address_bit(L.tslot[i]);
        for (int r = 0; r < ps->R; ++r) head.lreg[r] = ps->address_bit(L.rslot[r]);
        recs.clear();
        set_layout(L);
    }
    // the tile's lowest bits on lanes: the store writes whole runs
    bool storable() const {
        for (int s = 0; s < std::min(low_bits(dtype), ps->k); ++s)
            if (fn[s].reg != kNone || (fn[s].T & ~31u)) return false;
        return true;
    }
    int close(bool last) {
        if (last) flush_all();
        flush_phase();
        if (!storable()) emit_remap(make_layout(*ps, reg_slots() & ~((1u << std::min(low_bits(dtype), ps->k)) - 1u), true, dtype));
        for (int s = 0; s < ps->K; ++s) {
            const uint64_t ab = ps->address_bit(s);
            for (int i = 0; i < ps->NT; ++i)
                if ((fn[s].T >> i) & 1u) head.scol[i] ^= ab;
            if (fn[s].reg != kNone) head.sreg[fn[s].reg] ^= ab;
            if (fn[s].k) head.sconst ^= ab;
            if (fn[s].Q) head.soff[head.n_soff++] = {fn[s].Q, ab};
        }
        head.n_recs = (uint32_t)recs.size();
        return sink.launch(head, recs.data());
    }
    uint32_t reg_slots() const {
        uint32_t m = 0;
        for (int s = 0; s < ps->K; ++s)
            if (fn[s].reg != kNone) m |= 1u << s;
        return m;
    }
    void emit_sign_frame() {
        bool signs = false;
        for (uint32_t q = 0; q < 64; ++q) {
            const uint64_t later_q = q == 63 ? 0 : adj[q] & (~0ULL << (q + 1));
            if (later_q) {
                emit_sign(1ULL << q, later_q);
                signs = true;
            }
            adj[q] = 0;
        }
        if (zmask) {
            emit_sign(zmask, 0);
            signs = true;
            zmask = 0;
        }
        if (signs) rec(VM_FLUSHS);
    }
    // everything symbolic onto the amplitudes (end of the plan)
    void flush_all() {
        while (!terms.empty()) {
            apply_term(terms.back());
            terms.pop_back();
        }
        emit_sign_frame();
        if (scale.is_one()) return;
        if (!tph && scale.value().imag() == 0.0) {
            VmRec &w = rec(VM_SCALE);
            put(w.w + 4, 0, scale.value().real());
            scale = Scalar();
        } else {
            emit_scalar_phase();
        }
        flush_phase();
    }

    // the schedule's gates and remaps; cut: as many launches as the records need
    int emit_steps(const Sched &sc, bool cut) {
        later.assign(64, 0);
        for (const BGate &g : pass->gates) {
            const GClass c = class_of(g);
            if (c == G_DENSE || c == G_OVXY) ++later[g.q0];
        }
        bool z_open = false;
        for (const Step &st : sc.steps) {
            if (cut && (int)recs.size() + reserve() > kVmCapacity) {  // cut the launch; the next one loads the same registers
                const uint32_t keep = reg_slots();
                QF_TRY(close(false));
                open(make_layout(*ps, keep, true, dtype), true);
                z_open = false;
            }
            if (st.gate == kNone) {
                emit_remap(sc.layouts[st.layout]);
                z_open = false;
                continue;
            }
            const BGate &g = pass->gates[st.gate];
            const GClass c = class_of(g);
            switch (c) {
            case G_DENSE: emit_dense(g.q0, g.m, g.kraus); --later[g.q0]; break;
            case G_DIAG: emit_diag(g.q0, g.m, g.kraus); break;
            case G_ANTI: emit_anti(g.q0, g.m); break;
            case G_CNOT: emit_cnot(g.q0, g.q1); break;
            case G_CZ: toggle(g.q0, g.q1); break;
            case G_SWAP: emit_swap(g.q0, g.q1); std::swap(later[g.q0], later[g.q1]); break;
            case G_OVXY: emit_overlap_xy(g); --later[g.q0]; break;
            case G_OVZ: emit_overlap_z(g, !z_open); break;
            }
            z_open = c == G_OVZ;
            while (terms.size() > (size_t)kMaxTerms) {
                apply_term(terms.front());
                terms.erase(terms.begin());
            }
            // factors pulled out grow the stored amplitudes: bounded well inside float32's range
            if (scale.abs() < 0x1p-40) {  // a power of two: exact
                VmRec &w = rec(VM_SCALE);
                put(w.w + 4, 0, 0x1p-40);
                scale *= 0x1p40;
            }
        }
        return QF_OK;
    }

    int run(int R, int W) {
        for (size_t pi = 0; pi < plan.passes.size(); ++pi) {
            pass = &plan.passes[pi];
            const PassSlots slots(*pass, plan.n, R, W);
            ps = &slots;
            const auto sc = schedule(*pass, slots, plan.n, dtype);
            if (!sc) return fail(QF_ERR_INVALID_ARGUMENT, "register-tile pass could not be scheduled");
            open(sc->layouts[0], false);
            QF_TRY(emit_steps(*sc, true));
            QF_TRY(close(pi + 1 == plan.passes.size()));
        }
        return QF_OK;
    }
    // One unitary part of a trajectory program: from layout `from` to exactly
    // layout `to`, everything symbolic applied except the scalar: trajectories
    // carry unnormalised states, and a global phase means nothing to them. Its
    // magnitude tells how far the stored amplitudes have grown since their norm was
    // last brought near one. A run with state-dependent steps does that itself
    // (`measured`); otherwise it goes on to the next part, where emit_steps
    // takes 2^-40 out once it is due. (1024 Hadamards between two measured runs
    // would take the norm out of range.)
    int segment(const PassSlots &slots, const Pass &p, const Layout &from, const Layout &to, bool measured) {
        pass = &p;
        ps = &slots;
        set_layout(from);
        if (!p.gates.empty()) {
            const auto sc = schedule(p, slots, plan.n, dtype, &from);
            if (!sc) return fail(QF_ERR_INVALID_ARGUMENT, "register-tile segment could not be scheduled");
            QF_TRY(emit_steps(*sc, false));
        }
        later.assign(64, 0);
        apply_terms(false);  // on thread bits
        flush_phase_only();
        emit_sign_frame();
        if (!holds(to)) emit_remap(to);
        apply_terms(true);
        flush_phase_only();
        const double grown = scale.abs();
        scale = Scalar();
        if (!measured) scale *= grown;
        return QF_OK;
    }
    bool holds(const Layout &to) const {  // the amplitudes lie exactly as `to` has them
        for (int s = 0; s < ps->K; ++s)
            if (fn[s].k || fn[s].Q) return false;
        for (int i = 0; i < ps->NT; ++i)
            if (fn[(int)to.tslot[i]].T != 1u << i || fn[(int)to.tslot[i]].reg != kNone) return false;
        for (int r = 0; r < ps->R; ++r)
            if (fn[(int)to.rslot[r]].reg != r || fn[(int)to.rslot[r]].T) return false;
        return true;
    }
    void apply_terms(bool all) {
        for (size_t i = 0; i < terms.size();) {
            Fn r;
            if (!all && regs_of(terms[i].mask, &r)) {
                ++i;
                continue;
            }
            apply_term(terms[i]);
            terms.erase(terms.begin() + (long)i);
        }
    }
    void flush_phase_only() {
        if (tph) rec(VM_FLUSHP);
        tph = false;
    }

    // The records that one more step and the close of the launch can add: every
    // term, the sign frame, flushes, two remaps of up to eight records, a few gates.
    int reserve() const {
        if (recs.size() + kMaxTerms + 96 < (size_t)kVmCapacity) return 0;  // whatever it is
        int rows = 0;
        for (uint64_t m : adj) rows += m != 0;
        return (int)terms.size() + rows + 32;
    }
};

}  // namespace

// Decisions of a channel or measurement commute with gates on other qubits, so a
// gate joins the unitary part before the open run unless the run already acts
// on one of its qubits; a run holds one state-dependent step per qubit. Lists
// that the other engine refuses are left to it and its error texts.
int vm_lower_trajectories(uint32_t n, const qf_op *ops, uint64_t n_ops, TrajProgram &out, bool *ok) {
    *ok = false;
    out = TrajProgram();
    out.n = n;
    out.R = std::min(std::max((int)n, 6) - 5, 4);
    out.W = std::max((int)n, 6) - 5 - out.R;
    struct Part {
        std::vector<qf_op> gates, steps;
    };
    std::vector<Part> parts(1);
    uint64_t touched = 0, dependent = 0;
    for (uint64_t k = 0; k < n_ops; ++k) {
        const qf_op &o = ops[k];
        const bool gate = o.kind == QF_OP_GATE || o.kind == QF_OP_CNOT || o.kind == QF_OP_CZ || o.kind == QF_OP_SWAP;
        if (!gate && o.kind != QF_OP_CHANNEL && o.kind != QF_OP_MEASURE) return QF_OK;
        if (o.q0 >= n) return QF_OK;
        const bool decision = o.kind == QF_OP_CHANNEL || o.kind == QF_OP_MEASURE;
        uint64_t m = 1ULL << o.q0;
        if (o.kind == QF_OP_CNOT || o.kind == QF_OP_CZ || o.kind == QF_OP_SWAP) {
            if (o.q1 >= n || o.q1 == o.q0) return QF_OK;
            m |= 1ULL << o.q1;
        }
        const bool sd = decision && !(o.kind == QF_OP_CHANNEL && o.gate == QF_CHANNEL_DEPOLARIZING);
        if (decision ? (sd && (dependent & m)) : (touched & m) != 0) {
            parts.emplace_back();
            touched = dependent = 0;
        }
        if (decision) {
            parts.back().steps.push_back(o);
            touched |= m;
            if (sd) dependent |= m;
        } else {
            parts.back().gates.push_back(o);
        }
    }
    // trailing measurements of distinct qubits make a run of their own
    {
        std::vector<qf_op> &s = parts.back().steps;
        size_t t = s.size();
        while (t > 0 && s[t - 1].kind == QF_OP_MEASURE) --t;
        if (t > 0 && t < s.size()) {
            Part last;
            last.steps.assign(s.begin() + (long)t, s.end());
            s.resize(t);
            parts.push_back(std::move(last));
        }
    }
    std::vector<std::vector<BGate>> bound(parts.size());
    for (size_t i = 0; i < parts.size(); ++i)
        QF_TRY(bind_ops(n, parts[i].gates.data(), parts[i].gates.size(), nullptr, 0, nullptr, 0, -1, 0.0, bound[i]));
    while (!parts.empty() && parts.back().steps.empty()) parts.pop_back();  // gates that no decision follows
    Plan plan;
    plan.n = n;
    struct NoSink : VmSink {
        int launch(const VmHead &, const VmRec *) override { return QF_OK; }
    } none;
    Emitter e(plan, QF_C128, none);
    Layout at;
    for (size_t pi = 0; pi < parts.size(); ++pi) {
        const std::vector<BGate> &gates = bound[pi];
        Pass p;
        p.resident = (1ULL << n) - 1;
        if (!gates.empty()) {  // one-qubit runs merged; hundreds of these plans would push the searched ones out
            PlanOpts po;
            po.tile_qubits = po.low_qubits = (int)n;
            po.search = po.recorded = false;
            po.vm = po.merge_any = true;
            po.max_items = 1 << 30;
            Plan merged;
            QF_TRY(plan_passes(n, gates, po, merged));
            for (const Pass &x : merged.passes) p.gates.insert(p.gates.end(), x.gates.begin(), x.gates.end());
        }
        const PassSlots slots(p, n, out.R, out.W);
        // the run's layout
        const std::vector<qf_op> &st = parts[pi].steps;
        TrajRun r{};
        r.terminal = pi + 1 == parts.size();
        std::vector<int> order;  // state-dependent qubits in order
        for (const qf_op &o : st) {
            r.terminal = r.terminal && o.kind == QF_OP_MEASURE;
            if (!(o.kind == QF_OP_CHANNEL && o.gate == QF_CHANNEL_DEPOLARIZING)) order.push_back((int)o.q0);
        }
        r.n_sd = (uint32_t)order.size();
        uint32_t used = 0;
        Layout to;
        std::memset(&to, kNone, sizeof to);
        for (int q : order) used |= 1u << q;
        std::vector<int> all = order;
        for (int s = slots.K - 1; s >= 0; --s)
            if (!((used >> s) & 1u)) all.push_back(s);
        if (r.terminal) {  // first measured on the highest thread bit, the last ones on registers
            for (int i = 0; i < slots.NT; ++i) to.tslot[slots.NT - 1 - i] = (int8_t)all[i];
            for (int i = 0; i < slots.R; ++i) to.rslot[slots.R - 1 - i] = (int8_t)all[slots.NT + i];
        } else {  // the first state-dependent ones on register bits 0, 1, ...
            for (int i = 0; i < slots.R; ++i) to.rslot[i] = (int8_t)all[i];
            uint32_t rest = 0;
            for (int i = slots.R; i < slots.K; ++i) rest |= 1u << all[i];
            for (int s = 0, i = 0; s < slots.K; ++s)
                if ((rest >> s) & 1u) to.tslot[i++] = (int8_t)s;
        }
        if (pi == 0) {
            at = make_layout(slots, 0, true, QF_C128);
            for (int i = 0; i < slots.NT; ++i) out.lcol[i] = slots.address_bit(at.tslot[i]);
            for (int i = 0; i < slots.R; ++i) out.lreg[i] = slots.address_bit(at.rslot[i]);
        }
        r.rec_begin = (uint32_t)e.recs.size();
        QF_TRY(e.segment(slots, p, at, to, r.n_sd > 0));
        r.n_recs = (uint32_t)e.recs.size() - r.rec_begin;
        at = to;
        uint8_t pos[64];
        for (int i = 0; i < slots.NT; ++i) pos[(int)to.tslot[i]] = (uint8_t)(4 + i);
        for (int i = 0; i < slots.R; ++i) pos[(int)to.rslot[i]] = (uint8_t)i;
        r.step_begin = (uint32_t)out.steps.size();
        r.n_steps = (uint32_t)st.size();
        uint32_t n_sd = 0;
        for (size_t i = 0; i < st.size(); ++i) {
            const qf_op &o = st[i];
            TrajStep t{};
            t.pos = pos[o.q0];
            t.cbit = o.param;
            t.kind = TR_MEAS;
            if (o.kind == QF_OP_CHANNEL) {
                t.p = o.theta;
                if (!std::isfinite(t.p) || t.p < 0.0 || t.p > 1.0) return QF_OK;
                if (o.gate == QF_CHANNEL_THERMAL_DAMPING) {
                    const double beta = qf_op_aux(&o);
                    if (!std::isfinite(beta) || beta < 0.0) return QF_OK;
                    t.gu = t.p * std::exp(-beta);  // NoiseChannel::thermal_rates (src/lib.rs:1611-1626)
                }
                switch (o.gate) {
                case QF_CHANNEL_DEPOLARIZING: t.kind = TR_DEP; break;
                case QF_CHANNEL_AMPLITUDE_DAMPING: t.kind = TR_AD; break;
                case QF_CHANNEL_PHASE_DAMPING: t.kind = TR_PD; break;
                case QF_CHANNEL_THERMAL_DAMPING: t.kind = TR_TH; break;
                default: return QF_OK;
                }
                t.sp = std::sqrt(t.p);
                t.s1p = std::sqrt(1.0 - t.p);
                t.su = std::sqrt(t.gu);
                t.s1u = std::sqrt(1.0 - t.gu);
            }
            if (t.kind == TR_DEP) {
                for (size_t j = i + 1; j < st.size(); ++j)
                    if (st[j].q0 == o.q0 && !(st[j].kind == QF_OP_CHANNEL && st[j].gate == QF_CHANNEL_DEPOLARIZING)) t.later = 1;
            } else {
                t.sd = (uint8_t)n_sd++;
            }
            out.steps.push_back(t);
        }
        out.runs.push_back(r);
    }
    out.recs = std::move(e.recs);
    out.recs.emplace_back();  // the interpreter reads one head ahead
    *ok = !out.runs.empty();
    return QF_OK;
}

int vm_lower(const Plan &plan, int dtype, int R, int W, VmSink &sink) { return Emitter(plan, dtype, sink).run(R, W); }

int vm_run_f(qf_sv *psi, const Plan &plan);
int vm_run_d(qf_sv *psi, const Plan &plan);
int vm_run_d2(qf_sv *psi, qf_sv *lam, const Plan &plan, double *d_slot_sums);

int run_plan_vm(qf_sv *sv, const Plan &plan) { return sv->dtype == QF_C64 ? vm_run_f(sv, plan) : vm_run_d(sv, plan); }

int run_plan_vm_dual(qf_sv *psi, qf_sv *lam, const Plan &plan, double *d_slot_sums) {
    return vm_run_d2(psi, lam, plan, d_slot_sums);
}

}  // namespace qf
