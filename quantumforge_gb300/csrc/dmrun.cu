// dmrun.cu — runs of local channels on complex128 density matrices.
//
// A channel on qubit q acts on the (row bit n + q, column bit q) pair of every
// entry: v00' = a v00 + b v11, v11' = c v00 + d v11, v01' = e v01, v10' = f v10.
// One sweep per channel costs 2 to 3 FP64 operations per entry and real
// component and a launch (15 channels of a 10-qubit layer: 133 us, FP64 rate
// 1.7 lanes per clock and SM). Here a run of channels is first composed into one
// map per qubit (host), each map is split into shears and scales,
//   v00' = s00 (P0 + r0 Q0),  v11' = s11 (P1 + r1 Q1),  v01' = s01 v01,  v10' = s10 v10
// with P the entry of the larger coefficient of its row (so |r| <= 1), and the
// scales, which commute with the other qubits' maps, are all applied as one
// factor per entry by the last pass: 0.5 or 1 operations per entry and qubit
// plus 3 to 4 per entry in all. The 10-qubit layer then takes 41 us
// (16 and 24 us; 32 MB through L2 and 7 and 11 us of FP64 work).
//
// A pass holds a tile of 2^k entries, the (row, column) bits of up to (k - 2) / 2
// qubits and the two lowest column bits (64-byte runs); each thread keeps 2^RB
// of them in registers, the bit pairs of RB / 2 qubits at a time, and the tile
// changes hands through shared memory between qubits.
#include <algorithm>
#include <array>
#include <cmath>
#include <vector>

#include "qf_device.cuh"
#include "qf_internal.h"

namespace qf {

namespace {

constexpr int kRunRounds = 5;    // rounds of a pass
constexpr int kRunQubits = 17;   // of the matrix
constexpr uint32_t kRunThreads = 256;

struct ChannelRun {
    uint32_t n, k, n_rounds;
    uint32_t n_scale_tile, n_scale_thread;  // scales of qubits outside the tile, partly or wholly inside it
    uint64_t outer_mask, n_tiles;
    uint8_t tile_q[12];                     // matrix bit of each tile bit
    uint8_t reg[kRunRounds][4];             // tile bits of the register bits: column, row, column, row
    uint8_t thr[kRunRounds][8];             // tile bits of the thread index bits
    uint8_t flags[kRunRounds][2];           // 1: r0, 2: r1, 4: P0 = v11, 8: P1 = v00
    double r[kRunRounds][2][2];
    uint8_t scale_q[kRunQubits];            // tile's first, then threads'
    double scale[kRunQubits][4];            // by row bit << 1 | column bit
    double scale_reg[2][4];                 // qubits in the last round's registers
    uint32_t scaled;                        // the pass applies the scales
};

// 16-byte words, eight to a row of banks: bit b of the index moves bank bit b % 3
__device__ __forceinline__ uint32_t swz(uint32_t j) { return j ^ (((j >> 3) ^ (j >> 6) ^ (j >> 9)) & 7u); }

template <int RB, int SEL> __device__ __forceinline__ void mix(double2 (&v)[1 << RB], uint32_t flags, double r0, double r1) {
#pragma unroll
    for (int i = 0; i < (1 << RB); ++i) {
        if (i & (3 * SEL)) continue;
        const double2 x = v[i], y = v[i | (3 * SEL)];
        const double2 q0 = flags & 4 ? x : y, q1 = flags & 8 ? y : x;
        double2 p0 = flags & 4 ? y : x, p1 = flags & 8 ? x : y;
        if (flags & 1) {
            p0.x += r0 * q0.x;
            p0.y += r0 * q0.y;
        }
        if (flags & 2) {
            p1.x += r1 * q1.x;
            p1.y += r1 * q1.y;
        }
        v[i] = p0;
        v[i | (3 * SEL)] = p1;
    }
}

template <int RB>
__global__ void __launch_bounds__(kRunThreads, 2) k_dm_channel_run(double2 *__restrict__ rho, const __grid_constant__ ChannelRun a) {
    constexpr int E = 1 << RB;
    extern __shared__ __align__(16) unsigned char run_smem[];
    __shared__ double tile_scale[2];
    double2 *s = reinterpret_cast<double2 *>(run_smem);
    const uint32_t tid = threadIdx.x, nt = a.k - RB, last = a.n_rounds - 1;
    auto thread_index = [&](uint32_t r) {
        uint32_t j = 0;
        for (uint32_t b = 0; b < nt; ++b) j |= ((tid >> b) & 1u) << a.thr[r][b];
        return j;
    };
    auto matrix_bits = [&](uint32_t j) {
        uint64_t g = 0;
        for (uint32_t b = 0; b < a.k; ++b) g |= (uint64_t)((j >> b) & 1u) << a.tile_q[b];
        return g;
    };
    auto factor = [&](uint32_t i, uint64_t g) {
        return a.scale[i][((g >> (a.n + a.scale_q[i])) & 1ULL) << 1 | ((g >> a.scale_q[i]) & 1ULL)];
    };
    const uint64_t first_at = matrix_bits(thread_index(0)), last_at = matrix_bits(thread_index(last));
    uint32_t turn = 0;
    for (uint64_t t = blockIdx.x; t < a.n_tiles; t += gridDim.x, turn ^= 1u) {
        const uint64_t base = deposit(t, a.outer_mask);
        double2 v[E];
        {
            uint64_t m[RB];
#pragma unroll
            for (int b = 0; b < RB; ++b) m[b] = 1ULL << a.tile_q[a.reg[0][b]];
#pragma unroll
            for (int i = 0; i < E; ++i) {
                uint64_t g = base | first_at;
#pragma unroll
                for (int b = 0; b < RB; ++b)
                    if ((i >> b) & 1) g |= m[b];
                v[i] = rho[g];
            }
        }
        if (a.scaled && tid == 0) {
            double f = 1.0;
            for (uint32_t i = 0; i < a.n_scale_tile; ++i) f *= factor(i, base);
            tile_scale[turn] = f;
        }
        __syncthreads();  // the factor, and the last tile's reads of shared memory
        for (uint32_t r = 0;; ++r) {
            if (a.flags[r][0]) mix<RB, 1>(v, a.flags[r][0], a.r[r][0][0], a.r[r][0][1]);
            if constexpr (RB == 4)
                if (a.flags[r][1]) mix<RB, 4>(v, a.flags[r][1], a.r[r][1][0], a.r[r][1][1]);
            if (r == last) break;
#pragma unroll
            for (int p = 0; p < 2; ++p) {  // out in this round's order, back in the next one's
                const uint32_t at = swz(thread_index(r + p));
                uint32_t m[RB];
#pragma unroll
                for (int b = 0; b < RB; ++b) m[b] = swz(1u << a.reg[r + p][b]);
                if (p) __syncthreads();
#pragma unroll
                for (int i = 0; i < E; ++i) {
                    uint32_t j = at;
#pragma unroll
                    for (int b = 0; b < RB; ++b)
                        if ((i >> b) & 1) j ^= m[b];
                    if (p) v[i] = s[j];
                    else s[j] = v[i];
                }
            }
        }
        if (a.scaled) {
            double f = tile_scale[turn];
            for (uint32_t i = 0; i < a.n_scale_thread; ++i) f *= factor(a.n_scale_tile + i, base | last_at);
            double f0[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) f0[i] = f * a.scale_reg[0][i];
#pragma unroll
            for (int i = 0; i < E; ++i) {
                const double g = RB == 4 ? f0[i & 3] * a.scale_reg[1][i >> 2] : f0[i & 3];
                v[i] = make_double2(v[i].x * g, v[i].y * g);
            }
        }
        uint64_t m[RB];
#pragma unroll
        for (int b = 0; b < RB; ++b) m[b] = 1ULL << a.tile_q[a.reg[last][b]];
#pragma unroll
        for (int i = 0; i < E; ++i) {
            uint64_t g = base | last_at;
#pragma unroll
            for (int b = 0; b < RB; ++b)
                if ((i >> b) & 1) g |= m[b];
            rho[g] = v[i];
        }
    }
}

struct Split {  // one qubit's map: shears and scales
    uint32_t q;
    uint32_t flags = 0;
    double r[2], s[4];
};

Split split_map(uint32_t q, const double *k) {
    Split m;
    m.q = q;
    // row 0 over (v00, v11) with v00 preferred, row 1 with v11 preferred
    auto row = [](double own, double other, double &scale, double &ratio) {
        const bool swap = std::fabs(other) > std::fabs(own);
        scale = swap ? other : own;
        ratio = scale == 0.0 ? 0.0 : (swap ? own : other) / scale;
        return swap;
    };
    if (row(k[0], k[1], m.s[0], m.r[0])) m.flags |= 4;
    if (row(k[3], k[2], m.s[3], m.r[1])) m.flags |= 8;
    if (m.r[0] != 0.0) m.flags |= 1;
    if (m.r[1] != 0.0) m.flags |= 2;
    m.s[1] = k[4];
    m.s[2] = k[5];
    return m;
}

template <int RB> int launch_run(qf_sv *sv, const ChannelRun &a) {
    qf_ctx *ctx = sv->ctx;
    const size_t smem = sizeof(double2) << a.k;
    static size_t dyn[64] = {0};
    const int dev = ctx->device & 63;
    if (!dyn[dev]) QF_TRY(allow_max_dynamic_smem(k_dm_channel_run<RB>, ctx, &dyn[dev]));
    const uint32_t threads = 1u << (a.k - RB);
    int per_sm = 0;
    QF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_dm_channel_run<RB>, (int)threads, smem));
    const uint32_t grid = (uint32_t)std::min<uint64_t>(a.n_tiles, (uint64_t)std::max(per_sm, 1) * ctx->sm_count);
    k_dm_channel_run<RB><<<grid, threads, smem, ctx->stream>>>(static_cast<double2 *>(sv->d), a);
    QF_CUDA(cudaGetLastError());
    return QF_OK;
}

}  // namespace

int dm_channel_run(qf_sv *sv, uint32_t n, const uint32_t *qs, const double (*coefs)[6], size_t count) {
    if (sv->dtype != QF_C128 || n < 1 || n > (uint32_t)kRunQubits) return fail(QF_ERR_INVALID_ARGUMENT, "channel run on an unsupported matrix");
    // maps of one qubit compose; maps of different qubits commute
    std::array<std::array<double, 6>, kRunQubits> map;
    std::array<bool, kRunQubits> on{};
    for (size_t i = 0; i < count; ++i) {
        auto &m = map[qs[i]];
        const double *k = coefs[i];
        if (!on[qs[i]]) {
            std::copy(k, k + 6, m.begin());
            on[qs[i]] = true;
            continue;
        }
        const auto o = m;
        m = {k[0] * o[0] + k[1] * o[2], k[0] * o[1] + k[1] * o[3], k[2] * o[0] + k[3] * o[2], k[2] * o[1] + k[3] * o[3],
             k[4] * o[4], k[5] * o[5]};
    }
    std::vector<Split> maps;
    for (uint32_t q = 0; q < n; ++q)
        if (on[q]) maps.push_back(split_map(q, map[q].data()));
    if (maps.empty()) return QF_OK;
    if (maps.size() == 1) return dm_channel(sv, n, maps[0].q, map[maps[0].q].data());
    // Tile and registers: narrow tiles give small matrices more CTAs, four
    // entries a thread more warps; a tile of 12 bits (64 KB) pays only where it
    // saves a pass. Layer of 1.5 channels a qubit, with a pass of gates: 5 qubits
    // 15 us (10 tile bits: 19), 9 qubits 32 (16 entries a thread: 32, 8 bits:
    // 32), 10 qubits 54 with two passes of 12 bits (three of 10: 57, four
    // entries: 71), 11 qubits 156 with three of 10 (12 bits: 168).
    const uint32_t bits = 2 * n;
    const int rb = n <= 9 ? 2 : 4;
    const bool wide = rb == 4 && (maps.size() + 4) / 5 < (maps.size() + 3) / 4;
    const uint32_t k = std::min(bits, n <= 6 ? 8u : wide ? 12u : 10u);
    const size_t width = std::max<size_t>(1, (k - 2) / 2), passes = (maps.size() + width - 1) / width;
    for (size_t p = 0; p < passes; ++p) {
        const size_t b = maps.size() * p / passes, e = maps.size() * (p + 1) / passes, m = e - b;
        uint64_t mask = 3;
        for (size_t i = b; i < e; ++i) mask |= (1ULL << maps[i].q) | (1ULL << (n + maps[i].q));
        for (uint32_t c = 0; c < bits && (uint32_t)__builtin_popcountll(mask) < k; ++c) mask |= 1ULL << c;
        ChannelRun a{};
        a.n = n;
        a.k = (uint32_t)__builtin_popcountll(mask);
        a.outer_mask = ((1ULL << bits) - 1) & ~mask;
        a.n_tiles = 1ULL << (bits - a.k);
        uint8_t pos[2 * kRunQubits];
        uint32_t at = 0;
        for (uint32_t c = 0; c < bits; ++c)
            if ((mask >> c) & 1ULL) {
                a.tile_q[at] = (uint8_t)c;
                pos[c] = (uint8_t)at++;
            }
        // rounds: the highest qubits first, the lowest in between (their column
        // bits stay lane bits of the first and last round: longer runs)
        std::vector<std::array<size_t, 2>> rounds;  // maps in registers; a map that was done fills up
        std::vector<char> done(m, 0);
        auto add = [&](size_t x, size_t y) { rounds.push_back({b + x, b + y}); };
        if (rb == 2) {
            add(m - 1, m - 1);
            for (size_t i = 0; i + 1 < m; ++i) add(i, i);
        } else {
            add(m - 2, m - 1);
            for (size_t i = 0; i + 2 < m; i += 2) add(i, i + 1 < m - 2 ? i + 1 : m - 1);
        }
        a.n_rounds = (uint32_t)rounds.size();
        for (uint32_t r = 0; r < a.n_rounds; ++r) {
            uint32_t in_reg = 0;
            for (int c = 0; c < rb / 2; ++c) {
                const Split &sp = maps[rounds[r][c]];
                a.reg[r][2 * c] = pos[sp.q];
                a.reg[r][2 * c + 1] = pos[n + sp.q];
                in_reg |= (1u << pos[sp.q]) | (1u << pos[n + sp.q]);
                if (!done[rounds[r][c] - b]) {
                    a.flags[r][c] = (uint8_t)sp.flags;
                    a.r[r][c][0] = sp.r[0];
                    a.r[r][c][1] = sp.r[1];
                    done[rounds[r][c] - b] = 1;
                }
            }
            // thread bits in ascending order, but the first three on different bank bits
            uint32_t nt = 0, banks = 0;
            for (int step = 0; step < 2; ++step)
                for (uint32_t t = 0; t < a.k; ++t) {
                    if ((in_reg >> t) & 1u) continue;
                    if (step == 0 && ((banks >> (t % 3)) & 1u)) continue;
                    banks |= 1u << (t % 3);
                    in_reg |= 1u << t;
                    a.thr[r][nt++] = (uint8_t)t;
                }
        }
        if (p + 1 == passes) {
            a.scaled = 1;
            const auto &lastr = rounds.back();
            auto in_last = [&](size_t i) { return i == lastr[0] || (rb == 4 && i == lastr[1]); };
            for (int c = 0; c < rb / 2; ++c) std::copy(maps[lastr[c]].s, maps[lastr[c]].s + 4, a.scale_reg[c]);
            uint32_t ns = 0;
            for (int inside = 0; inside < 2; ++inside)
                for (size_t i = 0; i < maps.size(); ++i) {
                    const uint32_t q = maps[i].q;
                    const bool touches = ((mask >> q) & 1ULL) || ((mask >> (n + q)) & 1ULL);
                    if (in_last(i) || touches != (inside == 1)) continue;
                    a.scale_q[ns] = (uint8_t)q;
                    std::copy(maps[i].s, maps[i].s + 4, a.scale[ns]);
                    ++ns;
                    ++(inside ? a.n_scale_thread : a.n_scale_tile);
                }
        }
        if (rb == 4) QF_TRY(launch_run<4>(sv, a));
        else QF_TRY(launch_run<2>(sv, a));
    }
    return QF_OK;
}

}  // namespace qf
