// vmpass.cuh — the register-tile pass kernel (see vm.h), a template over the
// amplitude type, the register bits and whether lambda travels with psi.
//
// What bounds it. complex128: the FP64 pipe (1.7 lanes per clock and SM on
// GB300, 76 times below FP32), so a pass is priced by its FP64 instructions: two
// per amplitude for a dense gate, none for CNOTs, CZs, X/Y/Z gates and SWAPs
// (index and sign bookkeeping), four per thread for a phase on bits that a
// thread's registers share. A 25-qubit depth-40 circuit takes 1715 of them per
// amplitude and 104 ms, the pipe's rate (the shared-memory interpreter: 167 ms).
// complex64: instruction issue, a fifth of it arithmetic, so a 21-qubit depth-40
// circuit takes 0.54 ms (in-order register interpreter: 1.43 ms). Its kernel is
// held to 64 registers, 32 warps per SM, although that spills 40 bytes: at 96
// registers and 20 warps the circuit took 0.65 ms, at 80 and 24 0.58 ms.
#pragma once

#include <algorithm>

#include "vmexec.cuh"

namespace qf {
namespace vm {

template <typename C, int R, bool DUAL>
__global__ void __launch_bounds__(256, sizeof(C) == 8 && !DUAL ? 4 : 2)
    k_vm_pass(C *__restrict__ psi, C *__restrict__ lam, double *__restrict__ partials, uint32_t stride,
              const __grid_constant__ VmArgs a) {
    using T = typename Real<C>::T;
    using V = typename Reg<C>::T;
    using G = Reg<C>;
    using FP = File<C, 0>;
    using FL = File<C, 1>;
    constexpr int NR = 1 << R;
    FP::declare();
    if constexpr (DUAL) FL::declare();
    extern __shared__ __align__(16) unsigned char vm_smem[];
    const uint32_t tid = threadIdx.x, nthr = blockDim.x;
    const int nbits = 31 - __clz(nthr);
    V *buf = reinterpret_cast<V *>(vm_smem);
    V *bufl = buf + (DUAL ? (size_t)NR * nthr : 0);
    T *acc = reinterpret_cast<T *>(bufl + (size_t)NR * nthr);  // [warp][slot]
    if (DUAL) {
        const uint32_t n = a.h.n_ovl * (nthr >> 5);
        for (uint32_t s = tid; s < n; s += nthr) acc[s] = T(0);
        __syncthreads();
    }
    V *gp = reinterpret_cast<V *>(psi), *gl = reinterpret_cast<V *>(lam);
    uint64_t lbase = 0, sbase = a.h.sconst;
    for (int i = 0; i < nbits; ++i)
        if ((tid >> i) & 1u) {
            lbase ^= a.h.lcol[i];
            sbase ^= a.h.scol[i];
        }

    for (uint64_t t = blockIdx.x; t < a.h.n_tiles; t += gridDim.x) {
        const uint64_t tb = deposit(t, a.h.nonlocal_mask);
        const uint32_t tlo = (uint32_t)tb, thi = (uint32_t)(tb >> 32);
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            uint64_t ad = tb ^ lbase;
#pragma unroll
            for (int b = 0; b < R; ++b)
                if ((i >> b) & 1) ad ^= a.h.lreg[b];
            const bool in = ad < a.h.dim;
            FP::set(i, in ? gp[ad] : G::zero());
            if constexpr (DUAL) FL::set(i, in ? gl[ad] : G::zero());
        }
        vm_exec<C, R, DUAL>(a.recs, a.h.n_recs, tid, tlo, thi, buf, bufl, acc, a.h.n_ovl);
        uint64_t sb = tb ^ sbase;
        for (uint32_t k = 0; k < a.h.n_soff; ++k)
            if (__popcll(tb & a.h.soff[k].qm) & 1) sb ^= a.h.soff[k].col;
        __syncthreads();  // relabelled bits: a thread may store where another one of the CTA loaded
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            uint64_t ad = sb;
#pragma unroll
            for (int b = 0; b < R; ++b)
                if ((i >> b) & 1) ad ^= a.h.sreg[b];
            if (ad < a.h.dim) {
                gp[ad] = FP::get(i);
                if constexpr (DUAL) gl[ad] = FL::get(i);
            }
        }
    }
    if (DUAL) {
        __syncthreads();
        for (uint32_t s = tid; s < a.h.n_ovl; s += nthr) {
            double v = 0.0;
            for (uint32_t wv = 0; wv < (nthr >> 5); ++wv) v += acc[(size_t)wv * a.h.n_ovl + s];
            double *p = partials + (size_t)(a.h.slot_base + s) * stride + blockIdx.x;
            *p = a.h.accumulate ? *p + v : v;
        }
    }
}

inline size_t smem_bytes(size_t amp, int R, int W, bool dual, uint32_t n_ovl) {
    const size_t tile = amp << (5 + R + W);
    return (dual ? 2 * tile : tile) + (dual ? (size_t)8 * n_ovl << W : 0);
}

// Lowers the plan and launches its record streams on one grid; partials:
// [slot][grid].
template <typename C, int R, bool DUAL> struct Launcher : VmSink {
    qf_sv *psi, *lam;
    int threads;
    uint32_t grid = 0;
    size_t smem = 0;
    double *parts = nullptr;
    VmArgs args;

    int launch(const VmHead &h, const VmRec *recs) override {
        args.h = h;
        std::copy(recs, recs + h.n_recs, args.recs);
        qf_ctx *ctx = psi->ctx;
        k_vm_pass<C, R, DUAL><<<grid, threads, smem, ctx->stream>>>(static_cast<C *>(psi->d), DUAL ? static_cast<C *>(lam->d) : nullptr,
                                                                   parts, grid, args);
        QF_CUDA(cudaGetLastError());
        return QF_OK;
    }

    int run(const Plan &plan, int W, double *d_slot_sums) {
        qf_ctx *ctx = psi->ctx;
        threads = 32 << W;
        uint32_t max_ovl = 0;
        for (const Pass &p : plan.passes) max_ovl = std::max(max_ovl, p.a.n_slots);
        smem = smem_bytes(sizeof(C), R, W, DUAL, max_ovl);
        static size_t dyn[64] = {0};
        const int dev = ctx->device & 63;
        if (!dyn[dev]) QF_TRY(allow_max_dynamic_smem(k_vm_pass<C, R, DUAL>, ctx, &dyn[dev]));
        if (smem > dyn[dev])
            return fail(QF_ERR_UNSUPPORTED_OPERATION, "register-tile pass needs %zu bytes of shared memory (limit %zu)", smem,
                        dyn[dev]);
        const uint64_t tiles = plan.passes[0].a.n_tiles;
        if (tiles <= (uint64_t)ctx->sm_count) {
            grid = (uint32_t)tiles;
        } else {
            int per_sm = 0;
            QF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_vm_pass<C, R, DUAL>, threads, smem));
            grid = (uint32_t)std::min<uint64_t>((uint64_t)std::max(per_sm, 1) * ctx->sm_count, tiles);
        }
        if (DUAL && plan.n_slots) {
            QF_TRY(ensure_device(&ctx->ws_red, &ctx->ws_red_bytes, sizeof(double) * (size_t)plan.n_slots * grid));
            parts = static_cast<double *>(ctx->ws_red);
        }
        QF_TRY(vm_lower(plan, sizeof(C) == 8 ? QF_C64 : QF_C128, R, W, *this));
        if (DUAL && plan.n_slots) QF_TRY(reduce_slots(ctx, parts, grid, plan.n_slots, d_slot_sums));
        return QF_OK;
    }
};

template <typename C, int R, bool DUAL> int run_r(qf_sv *psi, qf_sv *lam, const Plan &plan, int W, double *d_slot_sums) {
    Launcher<C, R, DUAL> l;
    l.psi = psi;
    l.lam = lam;
    return l.run(plan, W, d_slot_sums);
}

template <typename C, bool DUAL> int run(qf_sv *psi, qf_sv *lam, const Plan &plan, double *d_slot_sums) {
    int R, W;
    vm_shape((int)plan.passes[0].a.k, sizeof(C) == 8 ? QF_C64 : QF_C128, DUAL, &R, &W);
    switch (R) {
    case 1: return run_r<C, 1, DUAL>(psi, lam, plan, W, d_slot_sums);
    case 2: return run_r<C, 2, DUAL>(psi, lam, plan, W, d_slot_sums);
    case 3: return run_r<C, 3, DUAL>(psi, lam, plan, W, d_slot_sums);
    default: break;
    }
    if constexpr (!DUAL) return run_r<C, 4, DUAL>(psi, lam, plan, W, d_slot_sums);
    return fail(QF_ERR_UNSUPPORTED_OPERATION, "register-tile pass: %d register bits", R);
}

}  // namespace vm

// The three instantiations, one translation unit each.
int vm_run_f(qf_sv *psi, const Plan &plan);
int vm_run_d(qf_sv *psi, const Plan &plan);
int vm_run_d2(qf_sv *psi, qf_sv *lam, const Plan &plan, double *d_slot_sums);

}  // namespace qf
