// dualpass.cu — backward adjoint passes of complex64 states below the compiled
// passes' size: psi and lambda of one tile in shared memory, the ops of the pass
// in order, as the shared-memory interpreter (sweep.cu) runs them and with its
// exact float32 operations, but in groups.
//
// What bounded the interpreter: one round trip of both tiles through shared
// memory and a barrier per gate, and two barriers with a double-precision tree
// per overlap (116 us for a 17-qubit pass of 96 gates and 41 overlaps on 32 CTAs;
// here 67 us). A group is a run of ops that one assignment of amplitudes to
// threads serves: its 2^R amplitudes of psi and of lambda per thread are read
// into registers once, every op of the group runs there, and they go back.
// The registers hold one bit b of 0..8 and the bits from 9 on, the thread index
// the others in order: with b = 8 gates and overlaps on the bits from 8 on and Z
// overlaps, with b < 8 gates and overlaps on b. These are the interpreter's own
// assignments (thread t takes the pairs t, t + 256, ...), so every thread's
// partial overlap sum is the same float. Signs (CZ) gather in a bit per amplitude
// and are applied before the next gate that mixes amplitudes. The
// partial sums wait in shared memory and are added 32 overlaps at a time, one
// warp each, in float32 with two levels of rounding errors carried along (72
// bits, the FP64 pipe being 76 times slower than the FP32 one).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "vmexec.cuh"

namespace qf {

namespace {

constexpr int kDualThreads = 256;
constexpr uint32_t kBatch = 32;  // overlaps whose partial sums wait together

constexpr uint8_t G_HIGH = 8, G_SHARED = 255;  // DualGroup::layout: the bit b, or no assignment
struct DualGroup {
    uint16_t begin, count;
    uint8_t layout;
    uint8_t pad[3];
};

__host__ __device__ inline uint32_t swz(uint32_t j) {  // float2 index; lanes 0..3 reach all four bank bits in every layout
    const uint32_t f = ((j >> 4) & 1u) * 15u ^ ((j >> 5) & 1u) * 5u ^ ((j >> 6) & 1u) * 6u ^ ((j >> 7) & 1u) * 9u ^
                       ((j >> 8) & 1u) * 3u ^ ((j >> 9) & 1u) * 10u ^ ((j >> 10) & 1u) * 12u ^ ((j >> 11) & 1u) * 7u;
    return j ^ f;
}

struct DualArgs {
    PassArgs pa;
    const TileOp *ops;
    const double *mats;
    const DualGroup *groups;
    uint32_t n_groups, stride;
};

struct DualSmem {
    uint32_t s0, s1, hi, ops, mats, groups, part, acc, total;
};
__host__ __device__ inline DualSmem dual_smem(const PassArgs &pa, uint32_t n_groups) {
    DualSmem L;
    uint32_t off = 0;
    auto take = [&](uint32_t bytes) {
        const uint32_t at = off;
        off += (bytes + 15) / 16 * 16;
        return at;
    };
    L.s0 = take(8u << pa.k);
    L.s1 = take(8u << pa.k);
    L.hi = take(8u << (pa.k - pa.low));
    L.ops = take((uint32_t)sizeof(TileOp) * pa.n_ops);
    L.mats = take(32 * pa.n_mats);
    L.groups = take((uint32_t)sizeof(DualGroup) * n_groups);
    L.part = take(4 * kDualThreads * kBatch);
    L.acc = take(8 * pa.n_slots);
    L.total = off;
    return L;
}

__device__ __forceinline__ uint32_t ones_of(int r) {  // amplitudes with register bit r set
    return r == 0 ? 0xAAAAu : r == 1 ? 0xCCCCu : r == 2 ? 0xF0F0u : 0xFF00u;
}
__device__ __forceinline__ uint32_t exchanged(uint32_t v, int r) {  // bit per amplitude, register bit r flipped
    const uint32_t hi = ones_of(r);
    return ((v & ~hi) << (1 << r)) | ((v & hi) >> (1 << r));
}

// cmac2 and cmul with each rounding where the interpreter has it: what the
// compiler contracts differs from kernel to kernel, so nothing is left to it
__device__ __forceinline__ float2 cmac2_rn(float2 m0, float2 a0, float2 m1, float2 a1) {
    float2 r;
    r.x = __fmaf_rn(-m1.y, a1.y, __fmaf_rn(m1.x, a1.x, __fmaf_rn(m0.x, a0.x, -__fmul_rn(m0.y, a0.y))));
    r.y = __fmaf_rn(m1.y, a1.x, __fmaf_rn(m1.x, a1.y, __fmaf_rn(m0.y, a0.x, __fmul_rn(m0.x, a0.y))));
    return r;
}
__device__ __forceinline__ float2 cmul_rn(float2 a, float2 f) {
    float2 r;
    r.x = __fmaf_rn(a.x, f.x, -__fmul_rn(a.y, f.y));
    r.y = __fmaf_rn(a.x, f.y, __fmul_rn(a.y, f.x));
    return r;
}
template <int B, int R, typename F> __device__ __forceinline__ void dense(float2 m00, float2 m01, float2 m10, float2 m11) {
#pragma unroll
    for (int i = 0; i < (1 << R); ++i)
        if (!((i >> B) & 1)) {
            const float2 a0 = vm::Reg<float2>::get(F::get(i)), a1 = vm::Reg<float2>::get(F::get(i | (1 << B)));
            F::set(i, vm::rpack(cmac2_rn(m00, a0, m01, a1)));
            F::set(i | (1 << B), vm::rpack(cmac2_rn(m10, a0, m11, a1)));
        }
}
template <int B, int R, typename F> __device__ __forceinline__ void cswap(bool c) {  // exchange where c
#pragma unroll
    for (int i = 0; i < (1 << R); ++i)
        if (!((i >> B) & 1)) {
            const auto x = F::get(i), y = F::get(i | (1 << B));
            F::set(i, c ? y : x);
            F::set(i | (1 << B), c ? x : y);
        }
}
template <int B, int R, typename F> __device__ __forceinline__ void diag(float2 d0, float2 d1) {
#pragma unroll
    for (int i = 0; i < (1 << R); ++i)
        F::set(i, vm::rpack(cmul_rn(vm::Reg<float2>::get(F::get(i)), B >= 0 && ((i >> (B & 3)) & 1) ? d1 : d0)));
}
// the interpreter's per-thread sum for Z, amplitudes in ascending order; `last`: the last amplitude's term
template <int B, int R> __device__ __forceinline__ float overlap_z(bool wide, float &last) {
    float sum = 0;
#pragma unroll
    for (int i = 0; i < (1 << R); ++i) {
        const float2 l = vm::Reg<float2>::get(vm::File<float2, 1>::get(i)), p = vm::Reg<float2>::get(vm::File<float2, 0>::get(i));
        const float v = __fmaf_rn(l.x, p.y, -__fmul_rn(l.y, p.x));
        last = B >= 0 && ((i >> (B & 3)) & 1) ? -v : v;
        if (wide || i == 0) sum += last;
    }
    return sum;
}
// the interpreter's per-thread sum, pairs in ascending order
template <int B, int R, bool Y> __device__ __forceinline__ float overlap_pairs() {
    using P = vm::File<float2, 0>;
    using L = vm::File<float2, 1>;
    using G = vm::Reg<float2>;
    float sum = 0;
#pragma unroll
    for (int i = 0; i < (1 << R); ++i)
        if (!((i >> B) & 1)) {
            const float2 l0 = G::get(L::get(i)), l1 = G::get(L::get(i | (1 << B)));
            const float2 p0 = G::get(P::get(i)), p1 = G::get(P::get(i | (1 << B)));
            if (!Y) {
                sum += __fadd_rn(__fmaf_rn(l0.x, p1.y, -__fmul_rn(l0.y, p1.x)), __fmaf_rn(l1.x, p0.y, -__fmul_rn(l1.y, p0.x)));
            } else {
                const float u = __fmaf_rn(l0.x, p1.x, __fmul_rn(l0.y, p1.y));
                const float v = __fmaf_rn(l1.x, p0.x, __fmul_rn(l1.y, p0.y));
                sum += __fsub_rn(v, u);
            }
        }
    return sum;
}

#define QF_DUAL_BITS(r, CALL)                                \
    switch (r) {                                             \
    case 0: CALL(0); break;                                  \
    case 1: if constexpr (R > 1) { CALL(1); } break;         \
    case 2: if constexpr (R > 2) { CALL(2); } break;         \
    default: if constexpr (R > 3) { CALL(3); } break;        \
    }

template <int R>
__global__ void __launch_bounds__(kDualThreads, 2)
    k_dual_pass(float2 *__restrict__ psi, float2 *__restrict__ lam, double *__restrict__ partials, const __grid_constant__ DualArgs a) {
    using FP = vm::File<float2, 0>;
    using FL = vm::File<float2, 1>;
    using G = vm::Reg<float2>;
    constexpr int NR = 1 << R;
    FP::declare();
    FL::declare();
    extern __shared__ __align__(16) unsigned char dual_buf[];
    const PassArgs &pa = a.pa;
    const DualSmem M = dual_smem(pa, a.n_groups);
    unsigned long long *s0 = reinterpret_cast<unsigned long long *>(dual_buf + M.s0);
    unsigned long long *s1 = reinterpret_cast<unsigned long long *>(dual_buf + M.s1);
    uint64_t *hi_off = reinterpret_cast<uint64_t *>(dual_buf + M.hi);
    TileOp *ops = reinterpret_cast<TileOp *>(dual_buf + M.ops);
    float2 *mats = reinterpret_cast<float2 *>(dual_buf + M.mats);
    DualGroup *groups = reinterpret_cast<DualGroup *>(dual_buf + M.groups);
    float *part = reinterpret_cast<float *>(dual_buf + M.part);
    double *acc = reinterpret_cast<double *>(dual_buf + M.acc);
    const uint32_t tid = threadIdx.x, T = 1u << pa.k, nhi = pa.k - pa.low, lowmask = (1u << pa.low) - 1;
    const bool wide = pa.k >= 9;              // every thread holds 2^R amplitudes
    const bool live = wide || tid < (T >> 1);  // else one pair, where there is one
    for (uint32_t h = tid; h < (1u << nhi); h += kDualThreads) {
        uint64_t off = 0;
        for (uint32_t r = 0; r < nhi; ++r)
            if ((h >> r) & 1u) off |= 1ULL << pa.hi_q[r];
        hi_off[h] = off;
    }
    for (uint32_t o = tid; o < pa.n_ops; o += kDualThreads) ops[o] = a.ops[o];
    for (uint32_t o = tid; o < a.n_groups; o += kDualThreads) groups[o] = a.groups[o];
    for (uint32_t e = tid; e < 4 * pa.n_mats; e += kDualThreads)
        mats[e] = make_float2((float)a.mats[2 * e], (float)a.mats[2 * e + 1]);
    for (uint32_t s = tid; s < pa.n_slots; s += kDualThreads) acc[s] = 0.0;
    __syncthreads();

    for (uint64_t t = blockIdx.x; t < pa.n_tiles; t += gridDim.x) {
        const uint64_t base = deposit(t, pa.nonlocal_mask);
        for (uint32_t v = tid; v < (T >> 1); v += kDualThreads) {
            const uint32_t j = v << 1;
            const uint64_t gi = base | hi_off[j >> pa.low] | (j & lowmask);
            const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(psi + gi), y = *reinterpret_cast<const ulonglong2 *>(lam + gi);
            s0[swz(j)] = x.x;
            s0[swz(j | 1u)] = x.y;
            s1[swz(j)] = y.x;
            s1[swz(j | 1u)] = y.y;
        }
        __syncthreads();
        uint32_t waiting = 0, first_slot = 0;  // overlaps with partial sums in `part`
        auto add_waiting = [&] {
            __syncthreads();
            const uint32_t lane = tid & 31u;
            for (uint32_t s = tid >> 5; s < waiting; s += kDualThreads / 32) {
                float h = 0.f, e = 0.f, f = 0.f;  // h + e + f: both levels of rounding errors are kept
                auto two = [](float &x, float y) {  // x += y; returns what rounding lost
                    const float t = x + y, yy = t - x;
                    const float lost = (x - (t - yy)) + (y - yy);
                    x = t;
                    return lost;
                };
                const float *row = part + s * kDualThreads;
                for (uint32_t j = lane; j < kDualThreads; j += 32) f += two(e, two(h, row[j]));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const float x = __shfl_xor_sync(0xffffffffu, h, o), xe = __shfl_xor_sync(0xffffffffu, e, o),
                                xf = __shfl_xor_sync(0xffffffffu, f, o);
                    const float l = two(h, x);
                    f += two(e, xe) + xf;
                    f += two(e, l);
                }
                double sum = (double)h + ((double)e + (double)f);
                if (__any_sync(0xffffffffu, !isfinite(h))) {  // a partial sum is not finite, or their float total is not
                    sum = 0.0;
                    for (uint32_t j = lane; j < kDualThreads; j += 32) sum += (double)row[j];
                    sum = warp_sum(sum);
                }
                if (lane == 0) acc[first_slot + s] += sum;
            }
            first_slot += waiting;
            waiting = 0;
            __syncthreads();
        };
        for (uint32_t gi = 0; gi < a.n_groups; ++gi) {
            const DualGroup g = groups[gi];
            if (g.layout == G_SHARED) {  // SWAP of two resident bits
                const TileOp op = ops[g.begin];
                const uint32_t lo = min(op.b0, op.b1), hi = max(op.b0, op.b1), m0 = 1u << op.b0, m1 = 1u << op.b1;
                for (uint32_t p = tid; p < (T >> 2); p += kDualThreads) {
                    const uint32_t b = insert00_32(p, lo, hi), i = swz(b | m1), j = swz(b | m0);
                    unsigned long long x = s0[i];
                    s0[i] = s0[j];
                    s0[j] = x;
                    x = s1[i];
                    s1[i] = s1[j];
                    s1[j] = x;
                }
                __syncthreads();
                continue;
            }
            // byte offsets of the thread's amplitudes (swz is linear over xor)
            const uint32_t b = g.layout, low = tid & ((1u << b) - 1u);
            const uint32_t at0 = swz(((tid ^ low) << 1) | low) << 3, at1 = at0 ^ (swz(1u << b) << 3);
            auto at = [&](int i) { return ((i & 1) ? at1 : at0) ^ (swz((uint32_t)(i >> 1) << 9) << 3); };
            if (live) {
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    const unsigned char *q = dual_buf + at(i);
                    FP::set(i, *reinterpret_cast<const unsigned long long *>(q + M.s0));
                    FL::set(i, *reinterpret_cast<const unsigned long long *>(q + M.s1));
                }
            }
            // where a tile bit lives: register bit or -1, and its value in the thread index
            auto reg_of = [&](uint32_t q) -> int { return q == b ? 0 : q >= 9 ? (int)q - 8 : -1; };
            auto bit_of = [&](uint32_t q) -> uint32_t { return (tid >> (q < b ? q : q - 1)) & 1u; };
            uint32_t signs = 0;  // amplitudes whose sign is still to be turned
            auto apply_signs = [&] {
                if (!__any_sync(0xffffffffu, signs)) return;
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    const uint32_t s = (signs << (31 - i)) & 0x80000000u;
                    FP::set(i, G::neg(FP::get(i), s));
                    FL::set(i, G::neg(FL::get(i), s));
                }
                signs = 0;
            };
            for (uint32_t o = g.begin; o < (uint32_t)g.begin + g.count; ++o) {
                const TileOp op = ops[o];
                const float2 *m = mats + 4 * op.mat;
                switch (op.kind) {
                case T_MAT1: {
                    apply_signs();
                    const float2 m00 = m[0], m01 = m[1], m10 = m[2], m11 = m[3];
#define QF_DUAL_DENSE(B)                           \
    dense<B, R, FP>(m00, m01, m10, m11);           \
    dense<B, R, FL>(m00, m01, m10, m11)
                    QF_DUAL_BITS(reg_of(op.b0), QF_DUAL_DENSE)
                    break;
                }
                case T_DIAG1:
                case T_GPHASE: {
                    const float2 d0 = m[0], d1 = m[3];
                    const int r = op.kind == T_DIAG1 ? reg_of(op.b0) : -1;
                    if (r >= 0) {
#define QF_DUAL_DIAG(B)       \
    diag<B, R, FP>(d0, d1);   \
    diag<B, R, FL>(d0, d1)
                        QF_DUAL_BITS(r, QF_DUAL_DIAG)
                        break;
                    }
                    const float2 f = (op.kind == T_DIAG1 ? bit_of(op.b0) != 0 : ((base >> op.g0) & 1ULL) != 0) ? d1 : d0;
                    if (op.kind == T_GPHASE && is_one(f)) break;
                    diag<-1, R, FP>(f, f);
                    diag<-1, R, FL>(f, f);
                    break;
                }
                case T_CNOT_LL:
                case T_CNOT_GL: {
                    const int rt = reg_of(op.b1), rc = op.kind == T_CNOT_LL ? reg_of(op.b0) : -1;
                    if (rc >= 0) {  // both in registers
                        const uint32_t moved = ones_of(rc);
                        signs = (signs & ~moved) | (exchanged(signs, rt) & moved);
#define QF_DUAL_CX(CB, TB)                                        \
    case 4 * CB + TB:                                             \
        if constexpr (R > CB && R > TB) {                         \
            vm::cx<CB, TB, R, FP>();                              \
            vm::cx<CB, TB, R, FL>();                              \
        }                                                         \
        break;
                        switch (4 * rc + rt) {
                            QF_DUAL_CX(0, 1) QF_DUAL_CX(0, 2) QF_DUAL_CX(0, 3) QF_DUAL_CX(1, 0) QF_DUAL_CX(1, 2) QF_DUAL_CX(1, 3)
                            QF_DUAL_CX(2, 0) QF_DUAL_CX(2, 1) QF_DUAL_CX(2, 3) QF_DUAL_CX(3, 0) QF_DUAL_CX(3, 1) QF_DUAL_CX(3, 2)
                        default: break;
                        }
                        break;
                    }
                    const bool c = op.kind == T_CNOT_LL ? bit_of(op.b0) != 0 : ((base >> op.g0) & 1ULL) != 0;
                    if (c) signs = exchanged(signs, rt);
#define QF_DUAL_CSWAP(B)     \
    cswap<B, R, FP>(c);      \
    cswap<B, R, FL>(c)
                    QF_DUAL_BITS(rt, QF_DUAL_CSWAP)
                    break;
                }
                case T_CZ_LL:
                case T_CZ_GL:
                case T_CZ_GG: {
                    uint32_t pat = 0xFFFFu;
                    auto with = [&](uint32_t q) {
                        const int r = reg_of(q);
                        pat &= r >= 0 ? ones_of(r) : bit_of(q) ? 0xFFFFu : 0u;
                    };
                    if (op.kind == T_CZ_LL) with(op.b0);
                    else if (!((base >> op.g0) & 1ULL)) pat = 0;
                    if (op.kind != T_CZ_GG) with(op.b1);
                    else if (!((base >> op.g1) & 1ULL)) pat = 0;
                    signs ^= pat;
                    break;
                }
                default: {  // overlaps
                    float sum = 0.f;
                    if (op.kind == T_OVL_X || op.kind == T_OVL_Y) {
                        apply_signs();
                        const bool y = op.kind == T_OVL_Y;
#define QF_DUAL_OVL(B) sum = y ? overlap_pairs<B, R, true>() : overlap_pairs<B, R, false>()
                        QF_DUAL_BITS(reg_of(op.b0), QF_DUAL_OVL)
                    } else {
                        // a sign that psi and lambda share drops out of their products
                        const int r = op.kind == T_OVL_ZL ? reg_of(op.b0) : -1;
                        const bool minus = op.kind == T_OVL_ZL ? r < 0 && bit_of(op.b0) : ((base >> op.g0) & 1ULL) != 0;
                        float last = 0.f;
#define QF_DUAL_OVLZ(B) sum = overlap_z<B, R>(wide, last)
                        if (r < 0) QF_DUAL_OVLZ(-1);
                        else QF_DUAL_BITS(r, QF_DUAL_OVLZ)
                        if (minus) {
                            sum = -sum;
                            last = -last;
                        }
                        // below 512 amplitudes each one is a sum of its own: the second of
                        // the pair takes the idle threads' place
                        if (!wide && tid < 128) part[waiting * kDualThreads + 128 + tid] = live ? last : 0.f;
                    }
                    const bool half = !wide && (op.kind == T_OVL_ZL || op.kind == T_OVL_ZG);
                    if (!half || tid < 128) part[waiting * kDualThreads + tid] = live ? sum : 0.f;
                    if (++waiting == kBatch) add_waiting();
                    break;
                }
                }
            }
            apply_signs();
            if (live) {
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    unsigned char *q = dual_buf + at(i);
                    *reinterpret_cast<unsigned long long *>(q + M.s0) = FP::get(i);
                    *reinterpret_cast<unsigned long long *>(q + M.s1) = FL::get(i);
                }
            }
            __syncthreads();
        }
        if (waiting) add_waiting();
        for (uint32_t v = tid; v < (T >> 1); v += kDualThreads) {
            const uint32_t j = v << 1;
            const uint64_t gi = base | hi_off[j >> pa.low] | (j & lowmask);
            *reinterpret_cast<ulonglong2 *>(psi + gi) = make_ulonglong2(s0[swz(j)], s0[swz(j | 1u)]);
            *reinterpret_cast<ulonglong2 *>(lam + gi) = make_ulonglong2(s1[swz(j)], s1[swz(j | 1u)]);
        }
        __syncthreads();
    }
    for (uint32_t s = tid; s < pa.n_slots; s += kDualThreads)
        partials[(size_t)(pa.slot_base + s) * a.stride + blockIdx.x] = acc[s];
}

// The pass's ops cut into groups, in order.
void group_ops(const TileOp *ops, uint32_t n_ops, uint32_t k, std::vector<DualGroup> &out) {
    const bool wide = k >= 9;
    // the layout an op needs: b, or -1 for any; `fits` tells whether a given one serves
    auto target = [&](const TileOp &op) -> int {
        if (op.kind == T_MAT1 || op.kind == T_OVL_X || op.kind == T_OVL_Y) return op.b0;
        if (op.kind == T_CNOT_LL || op.kind == T_CNOT_GL) return op.b1;
        return -1;
    };
    auto need = [&](const TileOp &op) -> int {
        if (op.kind == T_SWAP_LL) return G_SHARED;
        const int b = target(op);
        if (b >= 0) return wide && b >= 8 ? (int)G_HIGH : b;
        if (wide && (op.kind == T_OVL_ZL || op.kind == T_OVL_ZG)) return G_HIGH;
        return -1;
    };
    auto fits = [&](const TileOp &op, int layout) {
        const int nd = need(op);
        if (layout == G_SHARED || nd == G_SHARED) return false;
        if (nd < 0 || nd == layout) return true;
        // a gate on a bit from 9 on is in registers in every layout (overlap sums are not the same there)
        return wide && target(op) >= 9 && op.kind != T_OVL_X && op.kind != T_OVL_Y;
    };
    out.clear();
    for (uint32_t o = 0; o < n_ops;) {
        int layout = -1;
        for (uint32_t j = o; j < n_ops && layout < 0; ++j) layout = need(ops[j]);
        if (layout < 0) layout = wide ? (int)G_HIGH : 0;
        if (layout == G_SHARED && need(ops[o]) < 0) layout = wide ? (int)G_HIGH : 0;
        uint32_t e = o + 1;
        if (layout != G_SHARED)
            while (e < n_ops && fits(ops[e], layout)) ++e;
        DualGroup g{};
        g.begin = (uint16_t)o;
        g.count = (uint16_t)(e - o);
        g.layout = (uint8_t)layout;
        out.push_back(g);
        o = e;
    }
}

template <int R> int launch_dual(qf_sv *psi, qf_sv *lam, const Plan &plan, double *d_slot_sums) {
    qf_ctx *ctx = psi->ctx;
    static size_t dyn[64] = {0};
    const int dev = ctx->device & 63;
    if (!dyn[dev]) QF_TRY(allow_max_dynamic_smem(k_dual_pass<R>, ctx, &dyn[dev]));
    std::vector<std::vector<DualGroup>> groups(plan.passes.size());
    size_t n_groups = 0;
    uint32_t smem = 0;
    for (size_t i = 0; i < plan.passes.size(); ++i) {
        const Pass &p = plan.passes[i];
        group_ops(plan.ops.data() + p.op_begin, p.a.n_ops, p.a.k, groups[i]);
        n_groups += groups[i].size();
        smem = std::max(smem, dual_smem(p.a, (uint32_t)groups[i].size()).total);
    }
    if (smem > dyn[dev]) return run_plan_dual_smem(psi, lam, plan, d_slot_sums);
    std::vector<DualGroup> flat;
    flat.reserve(n_groups);
    for (const auto &g : groups) flat.insert(flat.end(), g.begin(), g.end());
    // one upload: ops, matrices, groups
    const size_t ops_n = plan.ops.size() * sizeof(TileOp), mats_n = plan.mats.size() * sizeof(double);
    const size_t ops_b = (ops_n + 15) / 16 * 16, mats_b = (mats_n + 15) / 16 * 16;
    std::vector<unsigned char> blob(ops_b + mats_b + n_groups * sizeof(DualGroup));
    std::memcpy(blob.data(), plan.ops.data(), ops_n);
    if (mats_n) std::memcpy(blob.data() + ops_b, plan.mats.data(), mats_n);
    size_t at = ops_b + mats_b;
    for (const auto &g : groups) {
        std::memcpy(blob.data() + at, g.data(), g.size() * sizeof(DualGroup));
        at += g.size() * sizeof(DualGroup);
    }
    QF_TRY(ensure_device(&ctx->ws_plan, &ctx->ws_plan_bytes, blob.size()));
    unsigned char *d = static_cast<unsigned char *>(ctx->ws_plan);
    QF_CUDA(cudaMemcpyAsync(d, blob.data(), blob.size(), cudaMemcpyHostToDevice, ctx->stream));
    int per_sm = 0;
    QF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_dual_pass<R>, kDualThreads, smem));
    const uint64_t tiles = plan.passes[0].a.n_tiles;
    const uint32_t grid = (uint32_t)std::min<uint64_t>((uint64_t)std::max(per_sm, 1) * ctx->sm_count, tiles);
    double *parts = nullptr;
    if (plan.n_slots) {
        QF_TRY(ensure_device(&ctx->ws_red, &ctx->ws_red_bytes, sizeof(double) * (size_t)plan.n_slots * grid));
        parts = static_cast<double *>(ctx->ws_red);
    }
    at = 0;
    for (size_t i = 0; i < plan.passes.size(); ++i) {
        const Pass &p = plan.passes[i];
        DualArgs a;
        a.pa = p.a;
        a.ops = reinterpret_cast<const TileOp *>(d) + p.op_begin;
        a.mats = reinterpret_cast<const double *>(d + ops_b) + 8 * (size_t)p.mat_begin;
        a.groups = reinterpret_cast<const DualGroup *>(d + ops_b + mats_b) + at;
        a.n_groups = (uint32_t)groups[i].size();
        a.stride = grid;
        at += groups[i].size();
        k_dual_pass<R><<<grid, kDualThreads, dual_smem(p.a, a.n_groups).total, ctx->stream>>>(
            static_cast<float2 *>(psi->d), static_cast<float2 *>(lam->d), parts, a);
        QF_CUDA(cudaGetLastError());
    }
    if (plan.n_slots) QF_TRY(reduce_slots(ctx, parts, grid, plan.n_slots, d_slot_sums));
    return QF_OK;
}

}  // namespace

int run_plan_dual_groups(qf_sv *psi, qf_sv *lam, const Plan &plan, double *d_slot_sums) {
    const uint32_t k = plan.passes[0].a.k;
    bool ok = k >= 2 && k <= 12;  // a pair per thread at least, 16 amplitudes at most
    for (const Pass &p : plan.passes) ok = ok && p.a.k == k && p.a.low >= 1 && p.a.n_ops > 0 && p.a.n_ops < 65536;
    for (const TileOp &t : plan.ops) ok = ok && t.kind <= T_OVL_ZG;
    if (!ok) return run_plan_dual_smem(psi, lam, plan, d_slot_sums);
    switch (k) {
    case 10: return launch_dual<2>(psi, lam, plan, d_slot_sums);
    case 11: return launch_dual<3>(psi, lam, plan, d_slot_sums);
    case 12: return launch_dual<4>(psi, lam, plan, d_slot_sums);
    default: return launch_dual<1>(psi, lam, plan, d_slot_sums);
    }
}

}  // namespace qf
