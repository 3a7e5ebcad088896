// vmexec.cuh — the record interpreter of the register-tile kernels (vm.h): the
// amplitudes' register files and the operations on them.
//
#pragma once



#include "qf_device.cuh"
#include "vm.h"

namespace qf {
namespace vm {

// The amplitudes of a thread live in PTX registers that only the inline asm
// below names (vr<i> for psi, vl<i> for lambda), not in C++ variables: an
// interpreter loop whose 50 branches all rewrite the array made the compiler copy
// the whole array on every record (60 % of the backward pass's instructions were
// moves). Every index is a constant after unrolling, so each access is one name;
// volatile asm keeps the accesses in order.
template <typename C> struct Reg;
template <> struct Reg<float2> {
    using T = unsigned long long;  // a packed pair, the operand of the packed FP32 instructions
    __device__ static __forceinline__ T pack(float x, float y) {
        T r;
        asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
        return r;
    }
    __device__ static __forceinline__ float2 get(T v) {
        float2 r;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
        return r;
    }
    __device__ static __forceinline__ T swap(T v) {
        const float2 a = get(v);
        return pack(a.y, a.x);
    }
    // a x + y with a given as a packed pair
    __device__ static __forceinline__ T fma2(T a, T x, T y) {
        T d;
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(x), "l"(y));
        return d;
    }
    __device__ static __forceinline__ T mul2(T a, T x) {
        T d;
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(x));
        return d;
    }
    __device__ static __forceinline__ T zero() { return 0ull; }
    __device__ static __forceinline__ T neg(T v, uint32_t s) { return v ^ (((T)s << 32) | s); }
};
template <> struct Reg<double2> {
    using T = double2;
    __device__ static __forceinline__ double2 get(T v) { return v; }
    __device__ static __forceinline__ T zero() { return make_double2(0.0, 0.0); }
    __device__ static __forceinline__ double flip(double v, uint32_t s) {
        return __hiloint2double(__double2hiint(v) ^ (int)s, __double2loint(v));
    }
    __device__ static __forceinline__ T neg(T v, uint32_t s) { return make_double2(flip(v.x, s), flip(v.y, s)); }
};

#define QF_VM_16(X) X(0) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15)
template <typename C, int A> struct File;  // A = 0: psi, 1: lambda
#define QF_VM_FILE(A, N)                                                                       \
    template <> struct File<float2, A> {                                                       \
        using V = unsigned long long;                                                          \
        __device__ static __forceinline__ void declare() { asm volatile(".reg .b64 " N "<16>;"); } \
        __device__ static __forceinline__ V get(int i) {                                       \
            V v = 0;                                                                           \
            switch (i) { QF_VM_16(QF_VM_GETF_##A) }                                            \
            return v;                                                                          \
        }                                                                                      \
        __device__ static __forceinline__ void set(int i, V v) {                               \
            switch (i) { QF_VM_16(QF_VM_SETF_##A) }                                            \
        }                                                                                      \
    };                                                                                         \
    template <> struct File<double2, A> {                                                      \
        using V = double2;                                                                     \
        __device__ static __forceinline__ void declare() {                                     \
            asm volatile(".reg .f64 " N "x<16>;");                                             \
            asm volatile(".reg .f64 " N "y<16>;");                                             \
        }                                                                                      \
        __device__ static __forceinline__ V get(int i) {                                       \
            V v = make_double2(0.0, 0.0);                                                      \
            switch (i) { QF_VM_16(QF_VM_GETD_##A) }                                            \
            return v;                                                                          \
        }                                                                                      \
        __device__ static __forceinline__ void set(int i, V v) {                               \
            switch (i) { QF_VM_16(QF_VM_SETD_##A) }                                            \
        }                                                                                      \
    };
#define QF_VM_GETF_0(i) case i: asm volatile("mov.b64 %0, vr" #i ";" : "=l"(v)); break;
#define QF_VM_SETF_0(i) case i: asm volatile("mov.b64 vr" #i ", %0;" ::"l"(v)); break;
#define QF_VM_GETD_0(i) case i: asm volatile("mov.f64 %0, vrx" #i "; mov.f64 %1, vry" #i ";" : "=d"(v.x), "=d"(v.y)); break;
#define QF_VM_SETD_0(i) case i: asm volatile("mov.f64 vrx" #i ", %0; mov.f64 vry" #i ", %1;" ::"d"(v.x), "d"(v.y)); break;
#define QF_VM_GETF_1(i) case i: asm volatile("mov.b64 %0, vl" #i ";" : "=l"(v)); break;
#define QF_VM_SETF_1(i) case i: asm volatile("mov.b64 vl" #i ", %0;" ::"l"(v)); break;
#define QF_VM_GETD_1(i) case i: asm volatile("mov.f64 %0, vlx" #i "; mov.f64 %1, vly" #i ";" : "=d"(v.x), "=d"(v.y)); break;
#define QF_VM_SETD_1(i) case i: asm volatile("mov.f64 vlx" #i ", %0; mov.f64 vly" #i ", %1;" ::"d"(v.x), "d"(v.y)); break;
QF_VM_FILE(0, "vr")
QF_VM_FILE(1, "vl")

__device__ __forceinline__ float flip_sign(float v, uint32_t s) { return __uint_as_float(__float_as_uint(v) ^ s); }
__device__ __forceinline__ double flip_sign(double v, uint32_t s) { return Reg<double2>::flip(v, s); }

template <typename C> struct Payload;
template <> struct Payload<float2> {
    static constexpr uint32_t kGenRecs = 1;
    __device__ static __forceinline__ float at(const uint32_t *w, int i) { return __uint_as_float(w[i]); }
};
template <> struct Payload<double2> {
    static constexpr uint32_t kGenRecs = 2;
    __device__ static __forceinline__ double at(const uint32_t *w, int i) {
        return __hiloint2double((int)w[2 * i + 1], (int)w[2 * i]);
    }
};

// x' = x + r0 y, y' = y + r1 x on register bit B, r real
template <int B, int R, typename F> __device__ __forceinline__ void fre(float r0, float r1) {
    using G = Reg<float2>;
    const unsigned long long p0 = G::pack(r0, r0), p1 = G::pack(r1, r1);
#pragma unroll
    for (int i = 0; i < (1 << R); ++i)
        if (!((i >> B) & 1)) {
            const unsigned long long x = F::get(i), y = F::get(i | (1 << B));
            F::set(i, G::fma2(p0, y, x));
            F::set(i | (1 << B), G::fma2(p1, x, y));
        }
}
template <int B, int R, typename F> __device__ __forceinline__ void fre(double r0, double r1) {
#pragma unroll
    for (int i = 0; i < (1 << R); ++i)
        if (!((i >> B) & 1)) {
            const double2 x = F::get(i), y = F::get(i | (1 << B));
            F::set(i, make_double2(fma(r0, y.x, x.x), fma(r0, y.y, x.y)));
            F::set(i | (1 << B), make_double2(fma(r1, x.x, y.x), fma(r1, x.y, y.y)));
        }
}
// the same with i r: i rho v = (-rho v.y, rho v.x)
template <int B, int R, typename F> __device__ __forceinline__ void fim(float r0, float r1) {
    using G = Reg<float2>;
#pragma unroll
    for (int i = 0; i < (1 << R); ++i)
        if (!((i >> B) & 1)) {
            const float2 x = G::get(F::get(i)), y = G::get(F::get(i | (1 << B)));
            F::set(i, G::pack(fmaf(-r0, y.y, x.x), fmaf(r0, y.x, x.y)));
            F::set(i | (1 << B), G::pack(fmaf(-r1, x.y, y.x), fmaf(r1, x.x, y.y)));
        }
}
template <int B, int R, typename F> __device__ __forceinline__ void fim(double r0, double r1) {
#pragma unroll
    for (int i = 0; i < (1 << R); ++i)
        if (!((i >> B) & 1)) {
            const double2 x = F::get(i), y = F::get(i | (1 << B));
            F::set(i, make_double2(fma(-r0, y.y, x.x), fma(r0, y.x, x.y)));
            F::set(i | (1 << B), make_double2(fma(-r1, x.y, y.x), fma(r1, x.x, y.y)));
        }
}
__device__ __forceinline__ unsigned long long rmul(unsigned long long v, float2 f) {
    const float2 a = Reg<float2>::get(v);
    return Reg<float2>::pack(a.x * f.x - a.y * f.y, a.x * f.y + a.y * f.x);
}
__device__ __forceinline__ double2 rmul(double2 v, double2 f) { return cmul(v, f); }
__device__ __forceinline__ unsigned long long rscale(unsigned long long v, float f) {
    return Reg<float2>::mul2(Reg<float2>::pack(f, f), v);
}
__device__ __forceinline__ double2 rscale(double2 v, double f) { return make_double2(v.x * f, v.y * f); }
__device__ __forceinline__ unsigned long long rpack(float2 v) { return Reg<float2>::pack(v.x, v.y); }
__device__ __forceinline__ double2 rpack(double2 v) { return v; }

template <int B, typename C, int R, typename F> __device__ __forceinline__ void gen(C m00, C m01, C m10, C m11) {
#pragma unroll
    for (int i = 0; i < (1 << R); ++i)
        if (!((i >> B) & 1)) {
            const C x = Reg<C>::get(F::get(i)), y = Reg<C>::get(F::get(i | (1 << B)));
            F::set(i, rpack(cmac2(m00, x, m01, y)));
            F::set(i | (1 << B), rpack(cmac2(m10, x, m11, y)));
        }
}
template <int CB, int TB, int R, typename F> __device__ __forceinline__ void cx() {
#pragma unroll
    for (int i = 0; i < (1 << R); ++i)
        if (((i >> CB) & 1) && !((i >> TB) & 1)) {
            const auto x = F::get(i), y = F::get(i | (1 << TB));
            F::set(i, y);
            F::set(i | (1 << TB), x);
        }
}
template <int A, int B, typename C, int R, typename F> __device__ __forceinline__ void neg2() {
#pragma unroll
    for (int i = 0; i < (1 << R); ++i)
        if (((i >> A) & 1) && ((i >> B) & 1)) F::set(i, Reg<C>::neg(F::get(i), 0x80000000u));
}
// sum over the thread's amplitudes of Im(conj(l) (P p)) for P = X or Y on register bit B
template <int B, bool Y, typename C, int R> __device__ __forceinline__ typename Real<C>::T ovl() {
    using P = File<C, 0>;
    using L = File<C, 1>;
    typename Real<C>::T s = 0, u = 0;
#pragma unroll
    for (int i = 0; i < (1 << R); ++i)
        if (!((i >> B) & 1)) {
            const C l0 = Reg<C>::get(L::get(i)), l1 = Reg<C>::get(L::get(i | (1 << B)));
            const C p0 = Reg<C>::get(P::get(i)), p1 = Reg<C>::get(P::get(i | (1 << B)));
            if (!Y) {
                s += l0.x * p1.y;
                u -= l0.y * p1.x;
                s += l1.x * p0.y;
                u -= l1.y * p0.x;
            } else {
                s -= l0.x * p1.x;
                u -= l0.y * p1.y;
                s += l1.x * p0.x;
                u += l1.y * p0.y;
            }
        }
    return s + u;
}

#define QF_VM_BITS(base, CALL)                                   \
    case (base): CALL(0); break;                                 \
    case (base) + 1: if constexpr (R > 1) { CALL(1); } break;    \
    case (base) + 2: if constexpr (R > 2) { CALL(2); } break;    \
    case (base) + 3: if constexpr (R > 3) { CALL(3); } break;

// Runs a record stream on the amplitudes in the register files. `buf` (and
// `bufl`): a tile each, for remaps; `acc`: overlap sums per warp and slot.
template <typename C, int R, bool DUAL>
__device__ __forceinline__ void vm_exec(const VmRec *recs, uint32_t n_recs, uint32_t tid, uint32_t tlo, uint32_t thi,
                                        typename Reg<C>::T *buf, typename Reg<C>::T *bufl, typename Real<C>::T *acc,
                                        uint32_t n_ovl) {
    using T = typename Real<C>::T;
    using PL = Payload<C>;
    using G = Reg<C>;
    using FP = File<C, 0>;
    using FL = File<C, 1>;
    constexpr int NR = 1 << R;
    auto sync = [] {
        if (blockDim.x > 32) __syncthreads();
        else __syncwarp();
    };
            C tph = mk(T(1), T(0));
            uint32_t smask = 0;
            T wt = 0, wz[R];  // Z-overlap sums: total, and with the sign of each register bit
#pragma unroll
            for (int b = 0; b < R; ++b) wz[b] = 0;

            // parity of a thread and tile mask
            auto par = [&](uint32_t tm, uint32_t q0, uint32_t q1) -> uint32_t {
                return __popc((tid & tm) ^ (tlo & q0) ^ (thi & q1)) & 1u;
            };
            // add a warp's sum of v to a slot
            auto slot_add = [&](T v, uint32_t slot) {
                v *= tph.x * tph.x + tph.y * tph.y;
                v = warp_sum(v);
                if ((tid & 31u) == 0) acc[(size_t)(tid >> 5) * n_ovl + slot] += v;
            };

            // the next record's head is fetched while the current one runs
            uint32_t head = recs[0].w[0];
            for (uint32_t o = 0; o < n_recs;) {
                const uint32_t kind = head & 0xFFu, on = o + ((head >> 8) & 0xFFu), flags = head >> 16;
                const uint32_t *w = recs[o].w;
                head = recs[on].w[0];
#define QF_VM_C1 par(w[2] & 0xFFFFu, w[8], w[9])
#define QF_VM_C2 par(w[2] >> 16, w[10], w[11])
                if (kind < 8) {
                    switch (kind) {
#define QF_VM_F(FN, B)                                          \
        {                                                           \
            T r0 = PL::at(w + 4, 0), r1 = PL::at(w + 4, 1);         \
            if (flags & 1u) { /* the thread sees the bit flipped */  \
                const bool e = QF_VM_C1;                            \
                const T s0 = e ? r1 : r0, s1 = e ? r0 : r1;         \
                r0 = s0;                                            \
                r1 = s1;                                            \
            }                                                       \
            if (flags & 2u) { /* and under a Z */                    \
                const uint32_t z = QF_VM_C2 << 31;                  \
                r0 = flip_sign(r0, z);                              \
                r1 = flip_sign(r1, z);                              \
            }                                                       \
            FN<B, R, FP>(r0, r1);                                   \
            if constexpr (DUAL) FN<B, R, FL>(r0, r1);               \
        }
#define QF_VM_FRE(B) QF_VM_F(fre, B)
#define QF_VM_FIM(B) QF_VM_F(fim, B)
                    QF_VM_BITS(VM_FRE, QF_VM_FRE)
                    QF_VM_BITS(VM_FIM, QF_VM_FIM)
                    default: break;
                    }
                } else if (kind < VM_GEN) {
                    switch (kind) {
#define QF_VM_PHASE(PAT)                                                            \
        {                                                                               \
            C f = mk(PL::at(w + 4, 0), PL::at(w + 4, 1));                               \
            if (flags && QF_VM_C1) { /* flipped bit: f goes to the others */     \
                tph = cmul(tph, f);                                                     \
                f.y = -f.y;                                                             \
            }                                                                           \
            _Pragma("unroll") for (int i = 0; i < NR; ++i) if (PAT) {                   \
                FP::set(i, rmul(FP::get(i), f));                                        \
                if constexpr (DUAL) FL::set(i, rmul(FL::get(i), f));                    \
            }                                                                           \
        }
#define QF_VM_DIAG(B) QF_VM_PHASE((i >> B) & 1)
                    QF_VM_BITS(VM_DIAG, QF_VM_DIAG)
                case VM_DIAGP: QF_VM_PHASE((w[1] >> i) & 1u) break;
                case VM_TPH:
                    if (QF_VM_C1 ^ flags) tph = cmul(tph, mk(PL::at(w + 4, 0), PL::at(w + 4, 1)));
                    break;
                case VM_FLUSHP:
#pragma unroll
                    for (int i = 0; i < NR; ++i) {
                        FP::set(i, rmul(FP::get(i), tph));
                        if constexpr (DUAL) FL::set(i, rmul(FL::get(i), tph));
                    }
                    tph = mk(T(1), T(0));
                    break;
                case VM_REMAP: {
                    const uint32_t *c = recs[o + 1].w;
                    uint32_t wb = w[6], rb = 0;
#pragma unroll
                    for (int i = 0; i < kVmMaxThreadBits; ++i)
                        if ((tid >> i) & 1u) {
                            wb ^= (c[i >> 1] >> (16 * (i & 1))) & 0xFFFFu;
                            rb ^= (c[4 + (i >> 1)] >> (16 * (i & 1))) & 0xFFFFu;
                        }
                    const uint32_t noff = w[1];
                    for (uint32_t k = 0; k < noff; ++k) {
                        const uint32_t *f = recs[o + 2 + (k >> 1)].w + 3 * (k & 1);
                        if (__popc((tlo & f[0]) ^ (thi & f[1])) & 1) wb ^= f[2];
                    }
                    sync();  // the previous remap's reads
#pragma unroll
                    for (int i = 0; i < NR; ++i) {
                        uint32_t j = wb;
#pragma unroll
                        for (int b = 0; b < R; ++b)
                            if ((i >> b) & 1) j ^= (w[2 + (b >> 1)] >> (16 * (b & 1))) & 0xFFFFu;
                        buf[j] = FP::get(i);
                        if constexpr (DUAL) bufl[j] = FL::get(i);
                    }
                    sync();
#pragma unroll
                    for (int i = 0; i < NR; ++i) {
                        uint32_t j = rb;
#pragma unroll
                        for (int b = 0; b < R; ++b)
                            if ((i >> b) & 1) j ^= (w[4 + (b >> 1)] >> (16 * (b & 1))) & 0xFFFFu;
                        FP::set(i, buf[j]);
                        if constexpr (DUAL) FL::set(i, bufl[j]);
                    }
                    break;
                }
                    default: break;
                    }
                } else {
                    switch (kind) {
#define QF_VM_GEN(B)                                                                  \
        {                                                                                 \
            const uint32_t *m = recs[o + 1].w, *n = recs[o + PL::kGenRecs].w;         \
            constexpr int h = PL::kGenRecs == 1 ? 4 : 0;                                  \
            C m00 = mk(PL::at(m, 0), PL::at(m, 1)), m01 = mk(PL::at(m, 2), PL::at(m, 3)); \
            C m10 = mk(PL::at(n, h), PL::at(n, h + 1)), m11 = mk(PL::at(n, h + 2), PL::at(n, h + 3)); \
            if (QF_VM_C1) {                                                               \
                C u = m00;                                                                \
                m00 = m11;                                                                \
                m11 = u;                                                                  \
                u = m01;                                                                  \
                m01 = m10;                                                                \
                m10 = u;                                                                  \
            }                                                                             \
            const uint32_t z = QF_VM_C2 << 31;                                            \
            m01 = mk(flip_sign(m01.x, z), flip_sign(m01.y, z));                           \
            m10 = mk(flip_sign(m10.x, z), flip_sign(m10.y, z));                           \
            gen<B, C, R, FP>(m00, m01, m10, m11);                                         \
            if constexpr (DUAL) gen<B, C, R, FL>(m00, m01, m10, m11);                     \
        }
                    QF_VM_BITS(VM_GEN, QF_VM_GEN)
#define QF_VM_CX(CB, TB)                             \
        case VM_CX + 4 * CB + TB:                        \
            if constexpr (R > CB && R > TB) {            \
                cx<CB, TB, R, FP>();                     \
                if constexpr (DUAL) cx<CB, TB, R, FL>(); \
            }                                            \
            break;
                    QF_VM_CX(0, 1) QF_VM_CX(0, 2) QF_VM_CX(0, 3) QF_VM_CX(1, 0) QF_VM_CX(1, 2) QF_VM_CX(1, 3)
                    QF_VM_CX(2, 0) QF_VM_CX(2, 1) QF_VM_CX(2, 3) QF_VM_CX(3, 0) QF_VM_CX(3, 1) QF_VM_CX(3, 2)
#define QF_VM_NEG(A, B)                                 \
        case VM_NEG + vm_pair(A, B):                        \
            if constexpr (R > B) {                          \
                neg2<A, B, C, R, FP>();                     \
                if constexpr (DUAL) neg2<A, B, C, R, FL>(); \
            }                                               \
            break;
                    QF_VM_NEG(0, 1) QF_VM_NEG(0, 2) QF_VM_NEG(1, 2) QF_VM_NEG(0, 3) QF_VM_NEG(1, 3) QF_VM_NEG(2, 3)
                case VM_TPH2: {
                    const uint32_t *m = recs[o + 1].w;
                    const bool e = (QF_VM_C1 ^ flags) != 0;
                    tph = cmul(tph, e ? mk(PL::at(m, 2), PL::at(m, 3)) : mk(PL::at(m, 0), PL::at(m, 1)));
                    break;
                }
                case VM_SGN:
                    smask ^= ((w[1] >> 16) ^ (QF_VM_C1 ? 0xFFFFu : 0u)) & ((w[1] & 0xFFFFu) ^ (QF_VM_C2 ? 0xFFFFu : 0u));
                    break;
                case VM_FLUSHS:
#pragma unroll
                    for (int i = 0; i < NR; ++i) {
                        const uint32_t s = (smask << (31 - i)) & 0x80000000u;
                        FP::set(i, G::neg(FP::get(i), s));
                        if constexpr (DUAL) FL::set(i, G::neg(FL::get(i), s));
                    }
                    smask = 0;
                    break;
                case VM_SCALE: {
                    const T f = PL::at(w + 4, 0);
#pragma unroll
                    for (int i = 0; i < NR; ++i) {
                        FP::set(i, rscale(FP::get(i), f));
                        if constexpr (DUAL) FL::set(i, rscale(FL::get(i), f));
                    }
                    break;
                }
#define QF_VM_OV(Y, B)                                          \
        if constexpr (DUAL) {                                       \
            T v = ovl<B, Y, C, R>() * PL::at(w + 4, 0);             \
            const uint32_t e = (Y ? QF_VM_C1 : 0u) ^ QF_VM_C2;      \
            slot_add(flip_sign(v, e << 31), w[1]);                  \
        }
#define QF_VM_OVX(B) QF_VM_OV(false, B)
#define QF_VM_OVY(B) QF_VM_OV(true, B)
                    QF_VM_BITS(VM_OVX, QF_VM_OVX)
                    QF_VM_BITS(VM_OVY, QF_VM_OVY)
                case VM_OVZ:
                    if constexpr (DUAL) {  // w_i = Im(conj(l_i) r_i); sums over halves give every register bit's sign sum
                        T x[NR];
#pragma unroll
                        for (int i = 0; i < NR; ++i) {
                            const C li = G::get(FL::get(i)), ri = G::get(FP::get(i));
                            x[i] = li.x * ri.y - li.y * ri.x;
                        }
#pragma unroll
                        for (int b = R - 1; b >= 0; --b) {
                            // fold register bit b: x[i] holds the sum over the bits above it; wz[b] its signed sum
                            T d = 0;
#pragma unroll
                            for (int i = 0; i < (1 << b); ++i) {
                                d += x[i] - x[i | (1 << b)];
                                x[i] += x[i | (1 << b)];
                            }
                            wz[b] = d;
                        }
                        wt = x[0];
                    }
                    break;
                case VM_OVZS:
                    if constexpr (DUAL) {
                        const uint32_t sel = w[1] >> 16;
                        T v = wt;
#pragma unroll
                        for (int b = 0; b < R; ++b)
                            if (sel == (uint32_t)b + 1) v = wz[b];
                        v *= PL::at(w + 4, 0);
                        slot_add(flip_sign(v, QF_VM_C1 << 31), w[1] & 0xFFFFu);
                    }
                    break;
                    default: break;
                    }
                }
                o = on;
            }
}

}  // namespace vm
}  // namespace qf
