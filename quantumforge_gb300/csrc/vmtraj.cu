// vmtraj.cu — noisy shots of small complex128 states (Circuit::run_shots_impl,
// src/lib.rs:2842-2916, with apply_channel_trajectory, src/lib.rs:1356-1506): one
// CTA per trajectory, its amplitudes in registers between the unitary record
// streams (vmexec.cuh) and the runs of random decisions (TrajRun).
//
// What bounds it: FP64 operations. Three things keep them few.
//  * A run of channels on distinct qubits needs only the populations |a|^2 and
//    the outcomes so far: with the outcomes assumed, every threshold of the run is
//    a partial sum of one contraction, and one block reduction returns all of
//    them. A shot whose draw falls the other way gives that step its outcome and
//    contracts again (rare: the assumed outcomes are the no-event ones). The
//    Kraus operators of the run are then one real factor per amplitude and an
//    index exchange. About 10 operations per amplitude and run, against 5.5 per
//    channel when each channel reduces P(1) and the norm and rescales the state.
//  * States stay unnormalised: a draw is compared as u N < p N, no division or
//    square root of a norm; powers of two keep the range, taken out behind every run
//    that finds the norm and, where none does, by the record streams.
//  * One trajectory is simulated once: the one on which no event happens, but for
//    the events that are certain. Every shot walks its own draws along that
//    trajectory's thresholds and starts from the snapshot at the run of its first
//    deviation; only what follows is its own.
// 20000 shots of a 12-qubit circuit with 4 noisy layers: 96.4 ms with every shot
// simulated gate by gate in shared memory, 8.5 ms here.
//
// Decisions equal the reference's except where a uniform lies within tie_eps of
// a threshold (counted); each shot draws from its own SmallRng position.
#include <algorithm>
#include <cstring>

#include "vmexec.cuh"

namespace qf {

namespace {

constexpr double kEps = 2.220446049250313e-16;
constexpr int kPos = 4 + kVmMaxThreadBits;
constexpr size_t kSnapshotBytes = size_t(64) << 20;

__device__ __forceinline__ double draw(uint64_t &x) {
    x ^= x << 13;
    x ^= x >> 7;
    x ^= x << 17;
    return (double)(x >> 11) * (1.0 / 9007199254740992.0);
}

// What the reference trajectory leaves for the shots.
struct TrajRef {
    double *p1, *norm;     // per step: P(1) and the norm before it, unnormalised (0 behind the trajectory's end)
    uint8_t *guess;        // per step: the outcome taken
    double2 *snapshots;    // amplitudes before every stride-th run, in the run's layout
    uint32_t stride;
};

struct TrajArgs {
    const VmRec *recs;
    const TrajRun *runs;
    const TrajStep *steps;
    uint32_t n_runs, n;
    TrajRef ref;
    uint64_t lcol[kVmMaxThreadBits], lreg[4];
    const double2 *init;
    uint64_t shots;
    uint32_t *first;              // per shot: the run it starts at (n_runs: none left)
    uint64_t *rng, *reg;          // per shot: generator and classical register there
    uint64_t *out;
    unsigned long long *ties, *next;
    int *err;
    double tie_eps;
    int share;                    // shots start from the reference trajectory's snapshots
};

// The outcome of one state-dependent step: population weights (w0, w1) and
// amplitude factors (f0, f1) of the ground and excited value, and whether the
// value flips.
struct Outcome {
    double w0, w1, f0, f1;
    int flip;
};
__device__ __forceinline__ Outcome outcome_of(const TrajStep &s, int o) {
    switch (s.kind) {
    case TR_AD: return o ? Outcome{0.0, s.p, 0.0, s.sp, 1} : Outcome{1.0, 1.0 - s.p, 1.0, s.s1p, 0};
    case TR_PD: return o ? Outcome{0.0, s.p, 0.0, s.sp, 0} : Outcome{1.0, 1.0 - s.p, 1.0, s.s1p, 0};
    case TR_TH:
        if (o == 1) return Outcome{0.0, s.p, 0.0, s.sp, 1};
        if (o == 2) return Outcome{s.gu, 0.0, s.su, 0.0, 1};
        return Outcome{1.0 - s.gu, 1.0 - s.p, s.s1u, s.s1p, 0};
    default: return o ? Outcome{0.0, 1.0, 0.0, 1.0, 0} : Outcome{1.0, 0.0, 1.0, 0.0, 0};
    }
}
// The outcome of step s at uniform u, P(1) and norm (unnormalised); *bn the norm
// of the branch taken.
__device__ __forceinline__ int decide(const TrajStep &s, double u, double p1, double norm, double tie_eps, double *bn,
                                      unsigned long long *ties) {
    const double un = u * norm, tie = tie_eps * norm;
    if (s.kind == TR_MEAS) {
        if (fabs(un - p1) < tie) ++*ties;
        const int o = un < p1 ? 1 : 0;
        *bn = o ? p1 : norm - p1;
        return o;
    }
    const double down = s.p * p1;
    if (s.kind != TR_TH) {
        if (fabs(un - down) < tie) ++*ties;
        const int o = un < down ? 1 : 0;
        *bn = o ? down : norm - down;
        return o;
    }
    const double up = s.gu * (norm - p1), du = down + up;
    if (fabs(un - down) < tie || fabs(un - du) < tie) ++*ties;
    const int o = un < down ? 1 : un < du ? 2 : 0;
    *bn = o == 1 ? down : o == 2 ? up : (norm - p1) * (1.0 - s.gu) + p1 * (1.0 - s.p);
    return o;
}
__device__ __forceinline__ bool bad_norm(double norm) { return !isfinite(norm) || norm <= 0.0; }
__device__ __forceinline__ bool bad_branch(double bn, double norm) { return !isfinite(bn) || bn <= kEps * norm; }
// the Pauli a depolarizing step applies (0, 1, 2), -1 for none (src/lib.rs:1369-1381)
__device__ __forceinline__ int pauli_of(const TrajStep &s, double u) {
    const double keep = __dsub_rn(1.0, s.p);
    if (!(u >= keep && s.p > 0.0)) return -1;
    const double b = floor(__dmul_rn(__dsub_rn(u, keep), __ddiv_rn(3.0, s.p)));
    return b >= 2.0 ? 2 : (int)b;
}

struct RunState {
    double w[kPos][2];       // state-dependent step j: population weights by the bit's value
    uint8_t pos[kPos], ex[kPos];  // its position and the value that counts as excited
    double sum[kPos + 1];    // reduced: norm, then P(1) of every state-dependent step
    double fac[kPos][2];     // per position: the run's amplitude factor by the bit's value
    uint8_t fl[kPos];        // and whether the bit has flipped
    double regf[16];
    uint32_t flip;           // position bits to exchange (thread bits, then register bits)
    int again, fault, trivial;
    uint64_t shot, rng, reg;
    uint32_t run;
};

// sums of the run's contraction under the assumed outcomes, into rs.sum
template <int R> __device__ __forceinline__ void contract(RunState &rs, uint32_t n_sd, double *red) {
    using FP = vm::File<double2, 0>;
    constexpr int NR = 1 << R;
    const uint32_t tid = threadIdx.x, nthr = blockDim.x;
    double w[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        const double2 a = FP::get(i);
        w[i] = a.x * a.x + a.y * a.y;
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < R; ++b) {  // register bit b: the b-th state-dependent qubit, or one that is summed out
        double odd = 0.0, even = 0.0;
        const bool step = (uint32_t)b < n_sd;
        if (step || b == 0) {
#pragma unroll
            for (int i = 0; i < NR; i += 2 << b) odd += w[i + (1 << b)];
            if (b == 0 || (step && rs.ex[b] == 0)) {
#pragma unroll
                for (int i = 0; i < NR; i += 2 << b) even += w[i];
            }
            if (b == 0) red[tid] = odd + even;
            if (step) red[(1 + b) * nthr + tid] = rs.ex[b] ? odd : even;
        }
        const double c0 = step ? rs.w[b][0] : 1.0, c1 = step ? rs.w[b][1] : 1.0;
#pragma unroll
        for (int i = 0; i < NR; i += 2 << b) w[i] = fma(c1, w[i + (1 << b)], c0 == 1.0 ? w[i] : c0 * w[i]);
    }
    double m = w[0];
    for (uint32_t j = R; j < n_sd; ++j) {
        const uint32_t x = (tid >> (rs.pos[j] - 4)) & 1u;
        red[(1 + j) * nthr + tid] = x == rs.ex[j] ? m : 0.0;
        m *= rs.w[j][x];
    }
    __syncthreads();
    for (uint32_t v = tid >> 5; v <= n_sd; v += nthr >> 5) {
        double s = 0.0;
        for (uint32_t i = tid & 31u; i < nthr; i += 32) s += red[v * nthr + i];
        s = warp_sum(s);
        if ((tid & 31u) == 0) rs.sum[v] = s;
    }
    __syncthreads();
}

// The reference trajectory's outcome of a state-dependent step: no event (the
// likelier result of a measurement), or an event where no event has no weight
// (damping of probability 1 on an excited qubit). *bn: the norm of that branch,
// without weight where every branch is (a state that is not finite).
__device__ __forceinline__ int reference_outcome(const TrajStep &s, double p1, double norm, double *bn) {
    if (s.kind == TR_MEAS) {
        const int o = p1 > 0.5 * norm ? 1 : 0;
        *bn = o ? p1 : norm - p1;
        return o;
    }
    unsigned long long t = 0;
    decide(s, 2.0, p1, norm, 0.0, bn, &t);  // above every threshold: no event
    if (!bad_branch(*bn, norm)) return 0;
    const double down = s.p * p1, up = s.kind == TR_TH ? s.gu * (norm - p1) : 0.0;
    *bn = down >= up ? down : up;
    return down >= up ? 1 : 2;
}

// One run of decisions on the amplitudes in the registers. REF: the reference
// trajectory (its outcomes recorded, no draws), else a shot. Returns false after a
// fault; the reference trajectory just ends there, as every shot leaves it at that
// step or before.
template <int R, bool REF>
__device__ __forceinline__ bool decide_run(const TrajArgs &a, RunState &rs, const TrajRun &run, double2 *buf) {
    using FP = vm::File<double2, 0>;
    using G = vm::Reg<double2>;
    constexpr int NR = 1 << R;
    const uint32_t tid = threadIdx.x, nthr = blockDim.x;
    double *red = reinterpret_cast<double *>(buf);
    const TrajStep *steps = a.steps + run.step_begin;
    for (uint32_t k = tid; k < (uint32_t)kPos; k += nthr) {
        rs.fac[k][0] = rs.fac[k][1] = 1.0;
        rs.fl[k] = 0;
    }
    for (uint32_t k = tid; k < run.n_steps; k += nthr)
        if (steps[k].kind != TR_DEP) {
            const uint32_t j = steps[k].sd;
            const Outcome o = outcome_of(steps[k], REF ? 0 : a.ref.guess[run.step_begin + k]);
            rs.w[j][0] = o.w0;
            rs.w[j][1] = o.w1;
            rs.pos[j] = steps[k].pos;
            rs.ex[j] = 1;
        }
    if (tid == 0) {
        rs.flip = 0;
        rs.fault = 0;
        rs.trivial = 1;
    }
    __syncthreads();
    uint32_t k0 = 0;
    double norm = 0.0;
    for (bool first = true;; first = false) {
        if (run.n_sd) contract<R>(rs, run.n_sd, red);
        if (tid == 0) {
            rs.again = 0;
            if (first) norm = run.n_sd ? rs.sum[0] : 1.0;
            if (bad_norm(norm)) rs.fault = 1;
            uint64_t x = rs.rng;
            unsigned long long ties = 0;
            uint32_t k = k0;
            for (; k < run.n_steps && !rs.fault && !rs.again; ++k) {
                const TrajStep s = steps[k];
                if (s.kind == TR_DEP) {
                    const int g = REF ? -1 : pauli_of(s, draw(x));
                    if (g < 0) continue;
                    const int e = rs.fl[s.pos] ^ 1;  // the bit value that is excited now
                    if (g >= 1) rs.fac[s.pos][e] = -rs.fac[s.pos][e];  // Y = i (-|0><1| + |1><0|), Z
                    if (g <= 1) {
                        rs.fl[s.pos] ^= 1;
                        rs.flip ^= 1u << s.pos;
                        if (s.later)
                            for (uint32_t j = k + 1; j < run.n_steps; ++j)
                                if (steps[j].kind != TR_DEP && steps[j].pos == s.pos) {
                                    const uint32_t d = steps[j].sd;
                                    rs.ex[d] ^= 1;
                                    const double t = rs.w[d][0];
                                    rs.w[d][0] = rs.w[d][1];
                                    rs.w[d][1] = t;
                                    rs.again = 1;
                                }
                    }
                    rs.trivial = 0;
                    continue;
                }
                const uint32_t j = s.sd;
                const double p1 = rs.sum[1 + j];
                int o, guess = REF ? 0 : a.ref.guess[run.step_begin + k];
                double bn;
                if (REF) {
                    a.ref.p1[run.step_begin + k] = p1;
                    a.ref.norm[run.step_begin + k] = norm;
                    o = reference_outcome(s, p1, norm, &bn);
                    a.ref.guess[run.step_begin + k] = (uint8_t)o;
                } else {
                    o = decide(s, draw(x), p1, norm, a.tie_eps, &bn, &ties);
                }
                if (bad_branch(bn, norm)) rs.fault = 1;
                norm = bn;
                const Outcome c = outcome_of(s, o);
                const int e = rs.ex[j];
                rs.fac[s.pos][e] *= c.f1;
                rs.fac[s.pos][e ^ 1] *= c.f0;
                if (c.flip) {
                    rs.fl[s.pos] ^= 1;
                    rs.flip ^= 1u << s.pos;
                }
                if (s.kind == TR_MEAS) rs.reg = (rs.reg & ~(1ULL << s.cbit)) | ((uint64_t)o << s.cbit);
                rs.trivial = 0;
                if (o != guess) {
                    rs.w[j][e] = c.w1;
                    rs.w[j][e ^ 1] = c.w0;
                    if (j + 1 < run.n_sd) rs.again = 1;
                }
            }
            k0 = k;
            rs.rng = x;
            if (ties) atomicAdd(a.ties, ties);
        }
        __syncthreads();
        if (rs.fault) {
            if (!REF && tid == 0) atomicExch(a.err, 1);
            return false;
        }
        if (!rs.again) break;
        __syncthreads();
    }
    if (rs.trivial) {
        __syncthreads();
        return true;
    }
    // one factor per amplitude; a power of two brings the norm back near one
    if (tid < NR) {
        int ex = 0;
        if (run.n_sd) frexp(rs.sum[0], &ex);
        double f = ldexp(1.0, -(ex >> 1));
        for (int b = 0; b < R; ++b) f *= rs.fac[b][(tid >> b) & 1u];
        rs.regf[tid] = f;
    }
    double f = 1.0;
    for (uint32_t t = 0; (1u << t) < nthr; ++t) f *= rs.fac[4 + t][(tid >> t) & 1u];
    __syncthreads();
    const uint32_t ftid = (rs.flip >> 4) & (nthr - 1), freg = rs.flip & (NR - 1);
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        const double g = f * rs.regf[i];
        const double2 v = FP::get(i);
        FP::set(i, make_double2(v.x * g, v.y * g));
    }
    if (rs.flip) {
#pragma unroll
        for (int i = 0; i < NR; ++i) buf[((uint32_t)i ^ freg) * nthr + (tid ^ ftid)] = FP::get(i);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NR; ++i) FP::set(i, buf[i * nthr + tid]);
    }
    __syncthreads();
    return true;
}

// Terminal measurements: the first one on the highest thread bit, the next ones
// below it, the last on register bits. A binary tree of partial sums answers
// every conditional probability; one thread descends.
template <int R>
__device__ __forceinline__ bool sample_run(const TrajArgs &a, RunState &rs, const TrajRun &run, double2 *buf) {
    using FP = vm::File<double2, 0>;
    constexpr int NR = 1 << R;
    const uint32_t tid = threadIdx.x, nthr = blockDim.x;
    double *heap = reinterpret_cast<double *>(buf);  // [1, 2 nthr)
    double *own = heap + 2 * nthr;                   // [thread][register]
    double w[NR], s = 0.0;
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        const double2 v = FP::get(i);
        w[i] = v.x * v.x + v.y * v.y;
        own[tid * NR + i] = w[i];
    }
#pragma unroll
    for (int h = NR / 2; h > 0; h >>= 1)
#pragma unroll
        for (int i = 0; i < NR / 2; ++i)
            if (i < h) w[i] += w[i + h];
    s = w[0];
    heap[nthr + tid] = s;
    __syncthreads();
    for (uint32_t h = nthr >> 1; h > 0; h >>= 1) {
        if (tid < h) heap[h + tid] = heap[2 * (h + tid)] + heap[2 * (h + tid) + 1];
        __syncthreads();
    }
    if (tid == 0) {
        rs.fault = 0;
        uint64_t x = rs.rng;
        unsigned long long ties = 0;
        uint32_t node = 1, base = 0, width = NR;
        double norm = heap[1];
        if (bad_norm(norm)) rs.fault = 1;
        for (uint32_t k = 0; k < run.n_steps && !rs.fault; ++k) {
            const TrajStep st = a.steps[run.step_begin + k];
            double p1;
            if (node < nthr) {
                p1 = heap[2 * node + 1];
            } else {
                width >>= 1;
                p1 = 0.0;
                for (uint32_t i = 0; i < width; ++i) p1 += own[(node - nthr) * NR + base + width + i];
            }
            double bn;
            const int o = decide(st, draw(x), p1, norm, a.tie_eps, &bn, &ties);
            if (bad_branch(bn, norm)) rs.fault = 1;
            rs.reg = (rs.reg & ~(1ULL << st.cbit)) | ((uint64_t)o << st.cbit);
            if (node < nthr) node = 2 * node + (uint32_t)o;
            else base += o ? width : 0;
            norm = bn;
        }
        if (ties) atomicAdd(a.ties, ties);
        if (rs.fault) atomicExch(a.err, 1);
    }
    __syncthreads();
    return rs.fault == 0;
}

template <int R, bool REF> __global__ void __launch_bounds__(256, 2) k_trajectory_runs(const __grid_constant__ TrajArgs a) {
    using FP = vm::File<double2, 0>;
    constexpr int NR = 1 << R;
    FP::declare();
    extern __shared__ __align__(16) unsigned char traj_buf[];
    double2 *buf = reinterpret_cast<double2 *>(traj_buf);
    __shared__ RunState rs;
    const uint32_t tid = threadIdx.x, nthr = blockDim.x;
    const size_t dim = (size_t)NR * nthr;
    for (;;) {
        __syncthreads();
        if (tid == 0) {
            if (REF) {
                rs.shot = 0;
                rs.run = 0;
            } else {  // the next shot with something left to do
                do {
                    rs.shot = atomicAdd(a.next, 1ULL);
                    if (rs.shot >= a.shots) break;
                    rs.run = a.share ? a.first[rs.shot] : 0;
                } while (rs.run >= a.n_runs);
                if (rs.shot < a.shots) {
                    rs.rng = a.rng[rs.shot];
                    rs.reg = a.share ? a.reg[rs.shot] : 0;
                }
            }
        }
        __syncthreads();
        const uint64_t shot = rs.shot;
        if (!REF && shot >= a.shots) return;
        uint32_t r = rs.run;
        const bool from_init = REF || !a.share;
        if (from_init) {
            uint64_t base = 0;
            for (uint32_t t = 0; (1u << t) < nthr; ++t)
                if ((tid >> t) & 1u) base |= a.lcol[t];
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                uint64_t ad = base;
#pragma unroll
                for (int b = 0; b < R; ++b)
                    if ((i >> b) & 1) ad |= a.lreg[b];
                FP::set(i, ad < (1ULL << a.n) ? a.init[ad] : make_double2(0.0, 0.0));
            }
        } else {
            const double2 *snap = a.ref.snapshots + (r / a.ref.stride) * dim;
#pragma unroll
            for (int i = 0; i < NR; ++i) FP::set(i, snap[i * nthr + tid]);
        }
        bool skip = !from_init;  // a snapshot is taken after the run's unitary part
        for (; r < a.n_runs; ++r) {
            const TrajRun run = a.runs[r];
            if (!skip) vm::vm_exec<double2, R, false>(a.recs + run.rec_begin, run.n_recs, tid, 0, 0, buf, nullptr, nullptr, 0);
            skip = false;
            __syncthreads();
            if (REF && r % a.ref.stride == 0) {
                double2 *snap = a.ref.snapshots + (r / a.ref.stride) * dim;
#pragma unroll
                for (int i = 0; i < NR; ++i) snap[i * nthr + tid] = FP::get(i);
            }
            if (run.terminal) {
                if (!REF && !sample_run<R>(a, rs, run, buf)) return;
                break;
            }
            if (!decide_run<R, REF>(a, rs, run, buf)) return;
        }
        if (REF) return;
        if (tid == 0) a.out[shot] = rs.reg;
    }
}

// Every shot along the reference trajectory until it leaves it.
__global__ void k_trajectory_first(const __grid_constant__ TrajArgs a) {
    for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < a.shots; s += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t x = a.rng[s], reg = 0, x0 = x, reg0 = 0;
        unsigned long long ties = 0, ties0 = 0;
        uint32_t start = 0, r = 0;
        bool event = false;
        for (; r < a.n_runs; ++r) {
            const TrajRun run = a.runs[r];
            if (r % a.ref.stride == 0) {
                start = r;
                x0 = x;
                reg0 = reg;
                ties0 = ties;
            }
            if (run.terminal) {
                event = true;
                break;
            }
            for (uint32_t k = run.step_begin; k < run.step_begin + run.n_steps && !event; ++k) {
                const TrajStep st = a.steps[k];
                const double u = draw(x);
                if (st.kind == TR_DEP) {
                    event = pauli_of(st, u) >= 0;
                    continue;
                }
                const double norm = a.ref.norm[k];
                double bn;
                const int o = decide(st, u, a.ref.p1[k], norm, a.tie_eps, &bn, &ties);
                event = o != a.ref.guess[k] || bad_norm(norm) || bad_branch(bn, norm);
                if (st.kind == TR_MEAS) reg = (reg & ~(1ULL << st.cbit)) | ((uint64_t)o << st.cbit);
            }
            if (event) break;
        }
        if (event) {  // the shot itself counts its ties from its first run on
            a.first[s] = start;
            a.rng[s] = x0;
            a.reg[s] = reg0;
            ties = ties0;
        } else {
            a.first[s] = a.n_runs;
            a.out[s] = reg;
        }
        if (ties) atomicAdd(a.ties, ties);
    }
}

template <int R> int launch(qf_ctx *ctx, TrajArgs &a, int W) {
    const int threads = 32 << W;
    const size_t dim = (size_t)threads << R;
    // a tile of amplitudes; the reductions and the sampling tree fit inside or beside it
    const size_t smem = std::max({dim * sizeof(double2), (size_t)(kPos + 1) * threads * sizeof(double),
                                  (2 * (size_t)threads + dim) * sizeof(double)});
    QF_CUDA(cudaFuncSetAttribute(k_trajectory_runs<R, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    QF_CUDA(cudaFuncSetAttribute(k_trajectory_runs<R, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    QF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trajectory_runs<R, false>, threads, smem));
    const uint64_t resident = (uint64_t)std::max(per_sm, 1) * ctx->sm_count, grid = std::min<uint64_t>(a.shots, resident);
    // When every shot has a CTA of its own at once, the reference trajectory would
    // only add its own time in front (134 shots of 6 qubits: 146 us with it, 118 without).
    a.share = a.shots > resident;
    if (a.share) {
        k_trajectory_runs<R, true><<<1, threads, smem, ctx->stream>>>(a);
        k_trajectory_first<<<(unsigned)std::min<uint64_t>((a.shots + 127) / 128, 8ull * ctx->sm_count), 128, 0, ctx->stream>>>(a);
    }
    k_trajectory_runs<R, false><<<(unsigned)grid, threads, smem, ctx->stream>>>(a);
    QF_CUDA(cudaGetLastError());
    return QF_OK;
}

}  // namespace

int run_trajectories_vm(qf_sv *init, const TrajProgram &prog, uint64_t shots, const uint64_t *starts, double tie_eps,
                        uint64_t *outcomes, uint64_t *n_ties) {
    qf_ctx *ctx = init->ctx;
    TrajArgs a;
    std::memset(&a, 0, sizeof a);
    a.n_runs = (uint32_t)prog.runs.size();
    a.n = prog.n;
    a.shots = shots;
    a.tie_eps = tie_eps;
    a.init = static_cast<const double2 *>(init->d);
    std::copy(prog.lcol, prog.lcol + kVmMaxThreadBits, a.lcol);
    std::copy(prog.lreg, prog.lreg + 4, a.lreg);
    const size_t snap = sizeof(double2) << (5 + prog.R + prog.W);
    const size_t most = std::max<size_t>(1, kSnapshotBytes / snap);
    a.ref.stride = (uint32_t)((a.n_runs + most - 1) / most);
    const size_t n_snap = (a.n_runs + a.ref.stride - 1) / a.ref.stride;
    const size_t n_steps = std::max<size_t>(prog.steps.size(), 1);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t at = off;
        off += (bytes + 255) / 256 * 256;
        return at;
    };
    const size_t o_recs = take(sizeof(VmRec) * prog.recs.size()), o_runs = take(sizeof(TrajRun) * prog.runs.size());
    const size_t o_steps = take(sizeof(TrajStep) * n_steps), o_p1 = take(8 * n_steps), o_norm = take(8 * n_steps);
    const size_t o_guess = take(n_steps), o_snap = take(snap * n_snap), o_first = take(4 * shots), o_rng = take(8 * shots);
    const size_t o_reg = take(8 * shots), o_out = take(8 * shots), o_cnt = take(32);
    QF_TRY(ensure_device(&ctx->ws_tree, &ctx->ws_tree_bytes, off));
    unsigned char *w = static_cast<unsigned char *>(ctx->ws_tree);
    a.recs = reinterpret_cast<const VmRec *>(w + o_recs);
    a.runs = reinterpret_cast<const TrajRun *>(w + o_runs);
    a.steps = reinterpret_cast<const TrajStep *>(w + o_steps);
    a.ref.p1 = reinterpret_cast<double *>(w + o_p1);
    a.ref.norm = reinterpret_cast<double *>(w + o_norm);
    a.ref.guess = w + o_guess;
    a.ref.snapshots = reinterpret_cast<double2 *>(w + o_snap);
    a.first = reinterpret_cast<uint32_t *>(w + o_first);
    a.rng = reinterpret_cast<uint64_t *>(w + o_rng);
    a.reg = reinterpret_cast<uint64_t *>(w + o_reg);
    a.out = reinterpret_cast<uint64_t *>(w + o_out);
    a.ties = reinterpret_cast<unsigned long long *>(w + o_cnt);
    a.next = a.ties + 1;
    a.err = reinterpret_cast<int *>(a.ties + 2);
    QF_CUDA(cudaMemcpyAsync(w + o_recs, prog.recs.data(), sizeof(VmRec) * prog.recs.size(), cudaMemcpyHostToDevice, ctx->stream));
    QF_CUDA(cudaMemcpyAsync(w + o_runs, prog.runs.data(), sizeof(TrajRun) * prog.runs.size(), cudaMemcpyHostToDevice, ctx->stream));
    QF_CUDA(cudaMemcpyAsync(w + o_steps, prog.steps.data(), sizeof(TrajStep) * prog.steps.size(), cudaMemcpyHostToDevice, ctx->stream));
    QF_CUDA(cudaMemcpyAsync(w + o_rng, starts, 8 * shots, cudaMemcpyHostToDevice, ctx->stream));
    QF_CUDA(cudaMemsetAsync(w + o_norm, 0, o_guess + n_steps - o_norm, ctx->stream));  // norms and outcomes
    QF_CUDA(cudaMemsetAsync(w + o_cnt, 0, 32, ctx->stream));
    switch (prog.R) {
    case 1: QF_TRY(launch<1>(ctx, a, prog.W)); break;
    case 2: QF_TRY(launch<2>(ctx, a, prog.W)); break;
    case 3: QF_TRY(launch<3>(ctx, a, prog.W)); break;
    default: QF_TRY(launch<4>(ctx, a, prog.W)); break;
    }
    if (outcomes) QF_CUDA(cudaMemcpyAsync(outcomes, a.out, 8 * shots, cudaMemcpyDeviceToHost, ctx->stream));
    QF_CUDA(cudaMemcpyAsync(ctx->h_small, a.ties, 32, cudaMemcpyDeviceToHost, ctx->stream));
    QF_CUDA(cudaStreamSynchronize(ctx->stream));
    unsigned long long t;
    int e;
    std::memcpy(&t, ctx->h_small, sizeof t);
    std::memcpy(&e, reinterpret_cast<unsigned char *>(ctx->h_small) + 16, sizeof e);
    if (e) return fail(QF_ERR_INVALID_PROBABILITY, "a shot selected a branch of probability <= f64::EPSILON");
    if (n_ties) *n_ties = t;
    return QF_OK;
}

}  // namespace qf
