// nb_direct.cu -- direct-sum gravity (K1) and the compensated kick-drift (K7).
//
// Replaces BruteForceCPU::Exec/Update (src/Sim/BruteForceCPU.cpp:25-74) and
// the D3D11 pair BruteForceGPU + shaders/Compute/Gravity.csh, Update.csh
// (src/Sim/BruteForceGPU.cpp:45-71).
//
// Layout: bodies are float4 (x, y, z, m) in HBM, padded to a multiple of
// kPad with zero-mass bodies.  Three force kernels:
//   * k_direct_pairs (large states): each unordered pair once, blocks taking
//     rows of 1024 targets against the source tiles behind them;
//   * k_direct_rows (small states): the same by single warps, rows of 128;
//   * k_direct_force (tuned handles, uncompensated sums): every interaction
//     from its target's side, BLOCK * IPT targets in registers against a
//     contiguous range of 128-body source tiles.
// The block kernels move source tiles (2 KB) from HBM to shared memory by the
// TMA engine (cp.async.bulk) into a double buffer guarded by mbarriers.  Forces
// are accumulated in FP32 in groups of sources, each group's sum folded into a
// compensated total.  K7 folds the partials in a fixed order (deterministic),
// applies G, and performs the kick-drift with Kahan-compensated velocity and
// position.
//
// Force law per source j on target i (reference law, Phys::Gravity,
// src/Sim/Physics.hpp:25-35, S = softening2):
//     a_i += m_j (p_j - p_i) / (r (r^2 + S)),   r = |p_j - p_i|
// evaluated with one MUFU.RSQ: 1/(r (r^2+S)) = rsqrt(r^2 (r^2+S)^2 + tiny).
// tiny = 1e-30 keeps the self pair (r = 0, dp = 0) finite, so it adds
// exactly zero; it is below the rounding of every real pair with S >= 1e-12.
// Plummer law: a_i += m_j (p_j - p_i) (r^2 + S)^{-3/2}.
#include "nb_common.cuh"
#include "nb_internal.hpp"
#include "nb_law.cuh"
#include "nb_pair_plan.hpp"
#include <algorithm>
#include <cmath>

namespace nb {

// K1: grid (target blocks, source ranges). Writes part[split][i] (sum) and
// part[splits + split][i] (compensation).  polls bounds each wait for a
// source tile (kMaxPolls normally; smaller only to test the timeout path);
// the copies still in flight after a wait gave up are always waited for with
// the full budget before the block exits.  HEAVY: the state's largest mass
// may need more than the law's default self-pair guard (masses above 1e21);
// the guard is then read from *mmax, else it is the compile-time constant.
template <int LAW, int BLOCK, int IPT, bool COMP, bool HEAVY>
__global__ void __launch_bounds__(BLOCK) k_direct_force(const float4* __restrict__ pos, int n_pad,
                                                        int tiles_per_split, int ntiles, int splits, float S,
                                                        float4* __restrict__ part, int* __restrict__ err,
                                                        uint32_t polls, const unsigned* __restrict__ mmax) {
    __shared__ __align__(128) float4 tile[2][kTileJ];
    const float tiny = HEAVY ? self_pair_tiny(mmax) : kTiny;
    __shared__ __align__(8) uint64_t bar[2];

    const int split = blockIdx.y;
    const int ibase = blockIdx.x * BLOCK * IPT + threadIdx.x;

    float xi[IPT], yi[IPT], zi[IPT];
    float sx[IPT], sy[IPT], sz[IPT], cx[IPT], cy[IPT], cz[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        float4 p = pos[ibase + k * BLOCK];
        xi[k] = p.x; yi[k] = p.y; zi[k] = p.z;
        sx[k] = sy[k] = sz[k] = 0.f;
        cx[k] = cy[k] = cz[k] = 0.f;
    }

    const int t_begin = split * tiles_per_split;
    const int nt = max(0, min(ntiles, t_begin + tiles_per_split) - t_begin);
    constexpr uint32_t kBytes = kTileJ * sizeof(float4);

    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 0; q < 2 && q < nt; ++q) {
            mbar_arrive_expect_tx(&bar[q], kBytes);
            bulk_g2s(tile[q], pos + (size_t)(t_begin + q) * kTileJ, kBytes, &bar[q]);
        }
    }

    int t = 0;
    bool abandoned = false;
    for (; t < nt; ++t) {
        const int b = t & 1;
        const bool ok = mbar_wait_bounded(&bar[b], (uint32_t)((t >> 1) & 1), polls);
        const float4* tj = tile[b];
#pragma unroll 1
        for (int f = 0; f < kTileJ; f += kFold) {
            float tx[IPT], ty[IPT], tz[IPT];
            if constexpr (IPT % 2 == 0) {
                // Packed FP32x2: target bodies (2k, 2k+1) share every instruction.
                constexpr int P = IPT / 2;
                float2 ax[P], ay[P], az[P];
#pragma unroll
                for (int k = 0; k < P; ++k) ax[k] = ay[k] = az[k] = make_float2(0.f, 0.f);
                const float2 S2 = make_float2(S, S), T2 = make_float2(tiny, tiny);
#pragma unroll 4
                for (int j = 0; j < kFold; ++j) {
                    const float4 pj = tj[f + j];
                    const float2 jx = make_float2(pj.x, pj.x), jy = make_float2(pj.y, pj.y);
                    const float2 jz = make_float2(pj.z, pj.z), jm = make_float2(pj.w, pj.w);
#pragma unroll
                    for (int k = 0; k < P; ++k)
                        interact_x2<LAW>(jx, jy, jz, jm, make_float2(-xi[2 * k], -xi[2 * k + 1]),
                                         make_float2(-yi[2 * k], -yi[2 * k + 1]), make_float2(-zi[2 * k], -zi[2 * k + 1]),
                                         S2, T2, ax[k], ay[k], az[k]);
                }
#pragma unroll
                for (int k = 0; k < P; ++k) {
                    tx[2 * k] = ax[k].x; tx[2 * k + 1] = ax[k].y;
                    ty[2 * k] = ay[k].x; ty[2 * k + 1] = ay[k].y;
                    tz[2 * k] = az[k].x; tz[2 * k + 1] = az[k].y;
                }
            } else {
#pragma unroll
                for (int k = 0; k < IPT; ++k) tx[k] = ty[k] = tz[k] = 0.f;
#pragma unroll 4
                for (int j = 0; j < kFold; ++j) {
                    const float4 pj = tj[f + j];
#pragma unroll
                    for (int k = 0; k < IPT; ++k)
                        interact<LAW>(pj, xi[k], yi[k], zi[k], S, tiny, tx[k], ty[k], tz[k]);
                }
            }
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                if (COMP) {
                    kahan_add(sx[k], cx[k], tx[k]);
                    kahan_add(sy[k], cy[k], ty[k]);
                    kahan_add(sz[k], cz[k], tz[k]);
                } else {
                    sx[k] += tx[k]; sy[k] += ty[k]; sz[k] += tz[k];
                }
            }
        }
        // Every thread is done with tile[b]; agree on the wait outcome.
        if (__syncthreads_or(!ok)) { abandoned = true; break; }
        if (threadIdx.x == 0 && t + 2 < nt) {
            fence_proxy_async_smem();
            mbar_arrive_expect_tx(&bar[b], kBytes);
            bulk_g2s(tile[b], pos + (size_t)(t_begin + t + 2) * kTileJ, kBytes, &bar[b]);
        }
    }
    if (abandoned) {
        // Let the copies still in flight land before the block's shared
        // memory is released (bounded), then report.
        if (threadIdx.x == 0) {
            for (int q = t; q < nt && q < t + 2; ++q)
                (void)mbar_wait_bounded(&bar[q & 1], (uint32_t)((q >> 1) & 1), kMaxPolls);
            record_error(err, DEV_WAIT_TIMEOUT);
        }
        return;
    }
    float4* psum = part + (size_t)split * n_pad;
    float4* pcmp = part + (size_t)(splits + split) * n_pad;
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int i = ibase + k * BLOCK;
        psum[i] = make_float4(sx[k], sy[k], sz[k], 0.f);
        pcmp[i] = make_float4(cx[k], cy[k], cz[k], 0.f);
    }
}

// K1 for large states: every unordered pair once (Newton's third law).
//
// The force kernel is bound by the FP32 pipe: 13 operations an interaction in
// k_direct_force.  A pair's separation and its reciprocal root serve both of
// its bodies, so doing the pair once costs 17 operations for two interactions.
//
// A row is a block of kPairRow = 1024 target bodies, eight a thread in
// registers (four packed FP32x2 pairs); a unit of work is a row against a run
// of source tiles at or after the row's own first tile.  Lane l of a warp
// takes source (l + r) mod 32 of a 32-body chunk at step r, read from the
// shared tile without bank conflicts, and the sources' own sums travel with
// them: six shuffles a step move them to the lane that takes that source
// next.  The four warps take the
// tile's four chunks in turn (a barrier between turns), adding the chunk's
// sums into the tile's shared totals in a fixed order, so results are
// deterministic.  Tiles of the row's own block take part as sources only: all
// their ordered pairs are evaluated from the target side.
//
// Targets are folded into compensated totals every FOLD sources (the totals
// live in shared memory, registers hold the running sums), sources every kPairGroup = 4 steps (16 terms in each packed half) into
// a second running sum and once a chunk into the totals.  A unit
// writes its targets' totals, and for each tile behind the row the sources':
// part holds kPairRow target partials per unit, then for each row of the launch
// one entry per body behind it.
// Bound by the FP32 pipe (77-79% of its cycles; three-operand packed
// instructions leave the rest).  Three blocks an SM at 156 registers: four
// (128) and five (102) measured 1% and 4% slower.  A step, GB300: 262,144
// bodies 28.5 -> 19.7 ms, 100,003 4.27 -> 2.97 ms, 20,001 217 -> 156 us; the
// force error against FP64 is k_direct_force's (2.8e-8 and 2.8e-8 at 262,144
// bodies of the Plummer sphere, 3.5e-8 and 3.5e-8 at 20,001).
constexpr int kPairThreads = 128, kPairIpt = 8, kPairGroup = 4;
static_assert(kPairRow == kPairThreads * kPairIpt && kPairRowTiles == kPairRow / kTileJ, "the planner's rows");
static_assert(kPairThreads == kTileJ, "one thread per source of a tile");
static_assert(kPad % kPairRow == 0, "padded states hold whole rows");

template <int LAW, bool HEAVY, int FOLD>
__global__ void __launch_bounds__(kPairThreads, kPairBlocksPerSm) k_direct_pairs(const float4* __restrict__ pos, int n_pad, int row0,
                                                                  int nrows, int per, float S,
                                                                  float4* __restrict__ part,
                                                                  int* __restrict__ err, uint32_t polls,
                                                                  const unsigned* __restrict__ mmax) {
    __shared__ __align__(128) float4 tile[2][kTileJ];
    __shared__ float tot[2][3 * kPairIpt][kPairThreads];   // targets: sums, compensations
    __shared__ float src[2][3][kTileJ];                    // the tile's sources: sums, compensations
    __shared__ __align__(8) uint64_t bar[2];
    // one block per unit and none empty: blocks that leave at once would still
    // take part in the first placement and leave some SMs with a unit more
    const int rows = n_pad / kPairRow, ntiles = n_pad / kTileJ, unit = blockIdx.x;
    int row = row0;
    for (int end = row0 + nrows; end - row > 1;) {   // the last row whose units start at or before this one
        const int mid = (row + end) / 2;
        if (pair_units_before(mid, row0, rows, per) <= unit) row = mid; else end = mid;
    }
    const int t_begin = row * kPairRowTiles + (unit - pair_units_before(row, row0, rows, per)) * per;
    const int nt = min(ntiles, t_begin + per) - t_begin;
    const float tiny = HEAVY ? self_pair_tiny(mmax) : kTiny;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int P = kPairIpt / 2;
    constexpr int kTurns = kTileJ / 32;
    constexpr uint32_t kBytes = kTileJ * sizeof(float4);
    const float2 S2 = make_float2(S, S), T2 = make_float2(tiny, tiny), z2 = make_float2(0.f, 0.f);

    float2 nx[P], ny[P], nz[P], mi[P];   // negated target coordinates, masses
#pragma unroll
    for (int q = 0; q < P; ++q) {
        const float4 a = pos[row * kPairRow + (2 * q) * kPairThreads + tid];
        const float4 b = pos[row * kPairRow + (2 * q + 1) * kPairThreads + tid];
        nx[q] = make_float2(-a.x, -b.x);
        ny[q] = make_float2(-a.y, -b.y);
        nz[q] = make_float2(-a.z, -b.z);
        mi[q] = make_float2(a.w, b.w);
    }
#pragma unroll
    for (int k = 0; k < 3 * kPairIpt; ++k) tot[0][k][tid] = tot[1][k][tid] = 0.f;
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (tid == 0) {
        for (int q = 0; q < 2 && q < nt; ++q) {
            mbar_arrive_expect_tx(&bar[q], kBytes);
            bulk_g2s(tile[q], pos + (size_t)(t_begin + q) * kTileJ, kBytes, &bar[q]);
        }
    }
    float4* sources = part + (size_t)gridDim.x * kPairRow + pair_source_base(row, row0, n_pad);
    auto fold_target = [&](int k, float x) {
        float s = tot[0][k][tid], c = tot[1][k][tid];
        kahan_add(s, c, x);
        tot[0][k][tid] = s;
        tot[1][k][tid] = c;
    };
    int t = 0;
    bool abandoned = false;
    for (; t < nt; ++t) {
        const float4* tj = tile[t & 1];
        const bool ok = mbar_wait_bounded(&bar[t & 1], (uint32_t)((t >> 1) & 1), polls);
        if (__syncthreads_or(!ok)) { abandoned = true; break; }
#pragma unroll 1
        for (int turn = 0; turn < kTurns; ++turn) {
            const int chunk = ((warp + turn) & (kTurns - 1)) * 32;
            float sx = 0.f, sy = 0.f, sz = 0.f;   // the travelling source's sums over whole groups of steps
#pragma unroll 1
            for (int h = 0; h < 32; h += FOLD) {
                float2 ax[P], ay[P], az[P];
#pragma unroll
                for (int q = 0; q < P; ++q) ax[q] = ay[q] = az[q] = z2;
#pragma unroll 1
                for (int g = h; g < h + FOLD; g += kPairGroup) {
                    float2 bx = z2, by = z2, bz = z2;
#pragma unroll
                    for (int u = 0; u < kPairGroup; ++u) {
                        const float4 pj = tj[chunk + ((lane + g + u) & 31)];
                        const float2 jx = make_float2(pj.x, pj.x), jy = make_float2(pj.y, pj.y);
                        const float2 jz = make_float2(pj.z, pj.z), jm = make_float2(pj.w, pj.w);
#pragma unroll
                        for (int q = 0; q < P; ++q) {
                            const float2 dx = __fadd2_rn(jx, nx[q]), dy = __fadd2_rn(jy, ny[q]), dz = __fadd2_rn(jz, nz[q]);
                            float2 wi, wj;
                            pair_factors_x2<LAW>(dx, dy, dz, S2, T2, jm, mi[q], wi, wj);
                            ax[q] = __ffma2_rn(wi, dx, ax[q]);
                            ay[q] = __ffma2_rn(wi, dy, ay[q]);
                            az[q] = __ffma2_rn(wi, dz, az[q]);
                            bx = __ffma2_rn(wj, dx, bx);
                            by = __ffma2_rn(wj, dy, by);
                            bz = __ffma2_rn(wj, dz, bz);
                        }
                        if (u + 1 < kPairGroup) {
                            const int next = (lane + 1) & 31;
                            bx.x = __shfl_sync(0xffffffffu, bx.x, next); bx.y = __shfl_sync(0xffffffffu, bx.y, next);
                            by.x = __shfl_sync(0xffffffffu, by.x, next); by.y = __shfl_sync(0xffffffffu, by.y, next);
                            bz.x = __shfl_sync(0xffffffffu, bz.x, next); bz.y = __shfl_sync(0xffffffffu, bz.y, next);
                        }
                    }
                    // this lane holds source (lane + g + kPairGroup - 1): its earlier groups' sums were left
                    // kPairGroup lanes on
                    const int from = (lane + kPairGroup) & 31;
                    sx = __shfl_sync(0xffffffffu, sx, from) + (bx.x + bx.y);
                    sy = __shfl_sync(0xffffffffu, sy, from) + (by.x + by.y);
                    sz = __shfl_sync(0xffffffffu, sz, from) + (bz.x + bz.y);
                }
#pragma unroll
                for (int q = 0; q < P; ++q) {
                    fold_target(6 * q, ax[q].x); fold_target(6 * q + 1, ay[q].x); fold_target(6 * q + 2, az[q].x);
                    fold_target(6 * q + 3, ax[q].y); fold_target(6 * q + 4, ay[q].y); fold_target(6 * q + 5, az[q].y);
                }
            }
            // lane l now holds source (l + 31) mod 32
            const float b[3] = {__shfl_sync(0xffffffffu, sx, (lane + 1) & 31), __shfl_sync(0xffffffffu, sy, (lane + 1) & 31),
                                __shfl_sync(0xffffffffu, sz, (lane + 1) & 31)};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                float s = turn == 0 ? 0.f : src[0][a][chunk + lane], c = turn == 0 ? 0.f : src[1][a][chunk + lane];
                kahan_add(s, c, b[a]);
                src[0][a][chunk + lane] = s;
                src[1][a][chunk + lane] = c;
            }
            __syncthreads();   // the next turn's warp continues this chunk's sums
        }
        // thread j owns source j from here to its own warp's next turn 0
        const int j = (t_begin + t) * kTileJ + tid;
        if (j >= (row + 1) * kPairRow)
            sources[j - (row + 1) * kPairRow] = make_float4(src[1][0][tid] - src[0][0][tid], src[1][1][tid] - src[0][1][tid],
                                                            src[1][2][tid] - src[0][2][tid], 0.f);
        if (tid == 0 && t + 2 < nt) {
            fence_proxy_async_smem();
            mbar_arrive_expect_tx(&bar[t & 1], kBytes);
            bulk_g2s(tile[t & 1], pos + (size_t)(t_begin + t + 2) * kTileJ, kBytes, &bar[t & 1]);
        }
    }
    if (abandoned) {
        // Let the copies still in flight land before the block's shared
        // memory is released (bounded), then report.
        if (tid == 0) {
            for (int q = t; q < nt && q < t + 2; ++q)
                (void)mbar_wait_bounded(&bar[q & 1], (uint32_t)((q >> 1) & 1), kMaxPolls);
            record_error(err, DEV_WAIT_TIMEOUT);
        }
        return;
    }
    float4* targets = part + (size_t)unit * kPairRow;
#pragma unroll
    for (int k = 0; k < kPairIpt; ++k)
        targets[k * kPairThreads + tid] = make_float4(tot[0][3 * k][tid] - tot[1][3 * k][tid],
                                                      tot[0][3 * k + 1][tid] - tot[1][3 * k + 1][tid],
                                                      tot[0][3 * k + 2][tid] - tot[1][3 * k + 2][tid], 0.f);
}

// K1 for small states: each pair once, by single warps.  A unit is a row of 128
// target bodies (four a lane) against up to L chunks of 32 sources behind it
// (direct_chunk; the row's own four chunks from the target side only), so that
// a few thousand bodies give a thousand warps of a few microseconds.  Bound by
// the FP32 pipe at a few warps a scheduler, and below some 2000 bodies by the
// latency of two dependent launches.  Those are programmatic dependent launches
// (nb_common.cuh), and a block is one warp, so that the units spread evenly.
// A step, with k_direct_force before: 1000 bodies 11.3 -> 6.7 us, 2048 12.3 ->
// 7.5, 4096 19.5 -> 12.5, 8192 45 -> 30; with ordinary launches 12.4, 12.4, 17.5
// and 37.  Early triggers (griddepcontrol.launch_dependents) gave nothing more, and
// in the update let the next step's warps gather on the SMs that emptied first
// (5000 bodies 32 us instead of 19).  Error against FP64 at 4096: 5.5e-8 (5.8e-8)
constexpr int kRowIpt = 4, kRowBodies = 32 * kRowIpt, kRowChunks = kRowBodies / kDirChunk;
struct RowPlan {
    int chunks, rows, per;   // source chunks, rows, chunks a unit (1, 2 or 4)
    __host__ __device__ int first_row_units() const { return (chunks + per - 1) / per; }
    // units of the rows before row r: row r has kRowChunks / per fewer than row r - 1
    __host__ __device__ int units_before(int r) const { return r * first_row_units() - (kRowChunks / per) * (r * (r - 1) / 2); }
    __host__ __device__ int row_units(int r) const { return first_row_units() - (kRowChunks / per) * r; }
};

// Entry of body (r + 1) * kRowBodies among row r's source partials (they follow
// the target partials, [units of a row][n_pad]).
__host__ __device__ inline size_t row_source_base(const RowPlan& p, int r, int n_pad) {
    return (size_t)p.first_row_units() * n_pad + (size_t)r * n_pad - (size_t)kRowBodies * (r * (r + 1) / 2);
}

template <int LAW>
__global__ void __launch_bounds__(32) k_direct_rows(const float4* pos, int n_pad, RowPlan plan, float S,
                                                                const unsigned* mmax, float4* part) {
    __shared__ float4 src[2][kDirChunk];
    const int lane = threadIdx.x, u = blockIdx.x;
    int row = -1;   // the last row whose units start at or before u
    for (int r0 = 0; r0 < plan.rows; r0 += 32)
        row += __popc(__ballot_sync(0xffffffffu, r0 + lane < plan.rows && plan.units_before(r0 + lane) <= u));
    const int s = u - plan.units_before(row);
    const int c0 = row * kRowChunks + s * plan.per, c1 = min(plan.chunks, c0 + plan.per);
    const int own = (row + 1) * kRowChunks;   // chunks before this one are the row's own
    wait_for_previous();
    const float tiny = mmax ? self_pair_tiny(mmax) : kTiny;
    const float2 S2 = make_float2(S, S), T2 = make_float2(tiny, tiny);
    constexpr int P = kRowIpt / 2;
    const int t0 = row * kRowBodies + lane;
    float2 nx[P], ny[P], nz[P], mi[P];
    float sum[3 * kRowIpt], comp[3 * kRowIpt];
    float4 cur = pos[c0 * kDirChunk + lane];
#pragma unroll
    for (int q = 0; q < P; ++q) {
        const float4 a = pos[t0 + (2 * q) * 32], b = pos[t0 + (2 * q + 1) * 32];
        nx[q] = make_float2(-a.x, -b.x);
        ny[q] = make_float2(-a.y, -b.y);
        nz[q] = make_float2(-a.z, -b.z);
        mi[q] = make_float2(a.w, b.w);
    }
#pragma unroll
    for (int k = 0; k < 3 * kRowIpt; ++k) sum[k] = comp[k] = 0.f;
    float4* sources = part + row_source_base(plan, row, n_pad);
    for (int c = c0; c < c1; ++c) {
        float4* buf = src[c & 1];
        buf[lane] = cur;
        __syncwarp();   // also: every lane is done with the chunk that this buffer held
        if (c + 1 < c1) cur = pos[(c + 1) * kDirChunk + lane];
        float3 f;
        if (c < own) {
            direct_chunk<LAW, kRowIpt, false>(buf, lane, nx, ny, nz, mi, S2, T2, sum, comp, f);
        } else {
            direct_chunk<LAW, kRowIpt, true>(buf, lane, nx, ny, nz, mi, S2, T2, sum, comp, f);
            sources[(c - own) * kDirChunk + lane] = make_float4(f.x, f.y, f.z, 0.f);
        }
    }
#pragma unroll
    for (int k = 0; k < kRowIpt; ++k)
        part[(size_t)s * n_pad + t0 + k * 32] =
            make_float4(sum[3 * k] - comp[3 * k], sum[3 * k + 1] - comp[3 * k + 1], sum[3 * k + 2] - comp[3 * k + 2], 0.f);
}

// K7: fold the partials of all source ranges (fixed order), apply G, add the
// pending initial forces, store the acceleration and, when update != 0,
// kick-drift: v += a dt; x += v dt / scale, both Kahan-compensated
// (src/Sim/BruteForceCPU.cpp:61-73).  When the error word is set (a force
// block abandoned a wait, or an earlier error has not been read yet) the
// step is abandoned: acceleration and state stay as they were.
// Render hand-off in the update's epilogue: the vertex (LWParticle layout,
// 32 bytes) of a body the update just moved, as two 16-byte stores.
__device__ __forceinline__ void write_vertex(nb_render_vertex* rv, const float4* rcol, float rscale, int i,
                                             const float4 x) {
    const float4 c = rcol[i];
    float4* o = reinterpret_cast<float4*>(rv + i);
    o[0] = make_float4(x.x, x.y, x.z, c.x);
    o[1] = make_float4(c.y, c.z, c.w, rscale);
}

// Body i's force from its source-split partials ([split][n_pad] sums, then
// [split][n_pad] compensations).
// kFoldLanes consecutive threads fold one body's partials: lane j takes
// splits j, j + kFoldLanes, ... (compensated, in that order), and the lanes'
// sums are added by a butterfly (every lane gets the same total).
__device__ __forceinline__ HiLo3 fold_partials_lanes(const float4* __restrict__ part, int splits, int n_pad, int i,
                                                      int j) {
    float ax = 0.f, ay = 0.f, az = 0.f, kx = 0.f, ky = 0.f, kz = 0.f, qx = 0.f, qy = 0.f, qz = 0.f;
    for (int s = j; s < splits; s += kFoldLanes) {
        const float4 p = part[(size_t)s * n_pad + i];
        const float4 c = part[(size_t)(splits + s) * n_pad + i];
        kahan_add(ax, kx, p.x);
        kahan_add(ay, ky, p.y);
        kahan_add(az, kz, p.z);
        qx += c.x; qy += c.y; qz += c.z;
    }
    return HiLo3{butterfly_total(ax, kx + qx), butterfly_total(ay, ky + qy), butterfly_total(az, kz + qz)};
}

// The same for k_direct_pairs' partials of rows [row0, row0 + rows): body i's
// target partials when its row is among them, and its entry as a source of
// each of those rows before its own.  A block's warps share 32 bodies (of one
// row), warp j taking every kFoldWarps-th entry; the first warp gets the totals.
// (Eight neighbouring threads a body: 10.6 us a fold at 50,001 bodies, now 8.9;
// the allocation-free call there 945 -> 937, a step of 262,144 20.10 -> 20.02 ms.)
__device__ __forceinline__ HiLo3 fold_pairs(const float4* __restrict__ part, const PairFold& pf, int n_pad, int i, int j,
                                            float (*sums)[6][32]) {
    float ax = 0.f, ay = 0.f, az = 0.f, kx = 0.f, ky = 0.f, kz = 0.f;
    const int row = i / kPairRow, last = pf.row0 + pf.rows, all = n_pad / kPairRow;
    auto add = [&](const float4 p) {
        kahan_add(ax, kx, p.x);
        kahan_add(ay, ky, p.y);
        kahan_add(az, kz, p.z);
    };
    if (row >= pf.row0 && row < last) {
        const int first = pair_units_before(row, pf.row0, all, pf.per);
        const int used = pair_units_before(row + 1, pf.row0, all, pf.per) - first;
        const float4* targets = part + (size_t)first * kPairRow + (i - row * kPairRow);
#pragma unroll 4
        for (int u = j; u < used; u += kFoldWarps) add(targets[(size_t)u * kPairRow]);
    }
    const float4* sources = part + (size_t)pair_units_before(last, pf.row0, all, pf.per) * kPairRow;
    const int end = min(row, last);
#pragma unroll 4
    for (int r = pf.row0 + j; r < end; r += kFoldWarps)
        add(sources[pair_source_base(r, pf.row0, n_pad) + (size_t)(i - (r + 1) * kPairRow)]);
    return add_warps(sums, ax, ay, az, kx, ky, kz);
}

// Adds a fold's total to a running (sum, low part); either may be the larger,
// which a Kahan addition does not allow for.
__device__ __forceinline__ void add_total(float& s, float& low, const HiLo& f) {
    float e;
    s = two_sum(s, f.hi, e);
    low += e + f.lo;
}

// Folds the partials of one of several launches of k_direct_pairs into the
// bodies' running (sum, low part); the first launch starts them.
__global__ void __launch_bounds__(32 * kFoldWarps) k_pairs_carry(const float4* __restrict__ part, PairFold pf, int n_pad, int first,
                              float4* __restrict__ carry, const int* __restrict__ err) {
    __shared__ float sums[kFoldWarps][6][32];
    const int i = blockIdx.x * 32 + (threadIdx.x & 31), j = threadIdx.x >> 5;
    if (*err != 0) return;
    const HiLo3 f = fold_pairs(part, pf, n_pad, i, j, sums);
    if (j != 0) return;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f), c = s;
    if (!first) {
        s = carry[i];
        c = carry[n_pad + i];
    }
    add_total(s.x, c.x, f.x); add_total(s.y, c.y, f.y); add_total(s.z, c.z, f.z);
    carry[i] = s;
    carry[n_pad + i] = c;
}

// The last launch's fold f plus what the earlier ones left in the carry (if any).
__device__ __forceinline__ float3 with_carry(const HiLo3& f, const float4* __restrict__ carry, int n_pad, int i) {
    if (!carry) return make_float3(f.x.rounded(), f.y.rounded(), f.z.rounded());
    float4 s = carry[i], c = carry[n_pad + i];
    add_total(s.x, c.x, f.x); add_total(s.y, c.y, f.y); add_total(s.z, c.z, f.z);
    return make_float3(s.x + c.x, s.y + c.y, s.z + c.z);
}

// What an update reads and writes (K7).
struct UpdateArgs {
    float G, dt, inv_scale;
    int update, comp;
    const float4* finit;
    float4 *acc, *pos, *posc, *vel, *velc;
    nb_render_vertex* rv;
    const float4* rcol;
    float rscale;
};

struct BodyState {
    float4 v, vc, x, xc;
    __device__ __forceinline__ void read(const UpdateArgs& u, int i) { v = u.vel[i]; vc = u.velc[i]; x = u.pos[i]; xc = u.posc[i]; }
};

__device__ __forceinline__ void finish_body(const UpdateArgs& u, int i, const float3 f, BodyState b) {
    float3 a = make_float3(u.G * f.x, u.G * f.y, u.G * f.z);
    if (u.finit) {
        const float4 f0 = u.finit[i];
        a.x += f0.x; a.y += f0.y; a.z += f0.z;
    }
    u.acc[i] = make_float4(a.x, a.y, a.z, 0.f);
    if (!u.update) return;
    float4 &v = b.v, &vc = b.vc, &x = b.x, &xc = b.xc;
    if (u.comp) {
        kahan_add(v.x, vc.x, a.x * u.dt);
        kahan_add(v.y, vc.y, a.y * u.dt);
        kahan_add(v.z, vc.z, a.z * u.dt);
        kahan_add(x.x, xc.x, ((v.x - vc.x) * u.dt) * u.inv_scale);
        kahan_add(x.y, xc.y, ((v.y - vc.y) * u.dt) * u.inv_scale);
        kahan_add(x.z, xc.z, ((v.z - vc.z) * u.dt) * u.inv_scale);
        u.velc[i] = vc;
        u.posc[i] = xc;
    } else {
        v.x += a.x * u.dt; v.y += a.y * u.dt; v.z += a.z * u.dt;
        x.x += (v.x * u.dt) * u.inv_scale; x.y += (v.y * u.dt) * u.inv_scale; x.z += (v.z * u.dt) * u.inv_scale;
    }
    u.vel[i] = v;
    u.pos[i] = x;
    if (u.rv) write_vertex(u.rv, u.rcol, u.rscale, i, x);
}

// After k_direct_force.
__global__ void k_direct_reduce_update(const float4* __restrict__ part, int splits, int n, int n_pad, UpdateArgs u,
                                       const int* __restrict__ err) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = t / kFoldLanes, j = t % kFoldLanes;
    // whole groups of lanes leave together (n_pad bodies, a multiple of the block)
    if (i >= n_pad || *err != 0) return;
    const HiLo3 total = fold_partials_lanes(part, splits, n_pad, i, j);
    if (i >= n || j != 0) return;
    BodyState b;
    b.read(u, i);
    finish_body(u, i, total.rounded(), b);
}

// After k_direct_pairs (carry: the earlier launches' sums, when there were several).
__global__ void __launch_bounds__(32 * kFoldWarps) k_direct_pairs_update(const float4* __restrict__ part, PairFold pf,
                                                                         const float4* __restrict__ carry, int n,
                                                                         int n_pad, UpdateArgs u,
                                                                         const int* __restrict__ err) {
    __shared__ float sums[kFoldWarps][6][32];
    const int i = blockIdx.x * 32 + (threadIdx.x & 31), j = threadIdx.x >> 5;
    if (*err != 0) return;
    const HiLo3 total = fold_pairs(part, pf, n_pad, i, j, sums);
    if (i >= n || j != 0) return;
    BodyState b;
    b.read(u, i);
    finish_body(u, i, with_carry(total, carry, n_pad, i), b);
}

// The fold of k_direct_rows' partials: a block's warps share 32 bodies, warp j
// taking every kFoldWarps-th partial of them.  Returns the force in the first
// warp's threads.
__device__ __forceinline__ float3 fold_rows(const float4* part, const RowPlan& plan, int n_pad, int i, int j,
                                            float (*sums)[6][32]) {
    float ax = 0.f, ay = 0.f, az = 0.f, kx = 0.f, ky = 0.f, kz = 0.f;
    const int row = i / kRowBodies;   // one row a block
    auto add = [&](const float4 p) {
        kahan_add(ax, kx, p.x);
        kahan_add(ay, ky, p.y);
        kahan_add(az, kz, p.z);
    };
    const int used = plan.row_units(row);
#pragma unroll 4
    for (int s = j; s < used; s += kFoldWarps) add(part[(size_t)s * n_pad + i]);
#pragma unroll 4
    for (int r = j; r < row; r += kFoldWarps) add(part[row_source_base(plan, r, n_pad) + (i - (r + 1) * kRowBodies)]);
    return add_warps(sums, ax, ay, az, kx, ky, kz).rounded();
}

__global__ void __launch_bounds__(32 * kFoldWarps) k_direct_rows_update(const float4* part, RowPlan plan, int n, int n_pad,
                                                                      UpdateArgs u, const int* err) {
    __shared__ float sums[kFoldWarps][6][32];
    const int i = blockIdx.x * 32 + (threadIdx.x & 31), j = threadIdx.x >> 5;
    wait_for_previous();
    const int failed = *err;
    BodyState b;
    if (j == 0) b.read(u, i);   // in flight beside the partials (i < n_pad)
    const float3 f = fold_rows(part, plan, n_pad, i, j, sums);
    if (j == 0 && i < n && failed == 0) finish_body(u, i, f, b);
}

// Kick-drift from a stored acceleration (Barnes-Hut path,
// src/Sim/BarnesHut.cpp:81-95).
__global__ void k_kick_drift(const float4* acc, int n, float4* pos,
                             float4* posc, float4* vel, float4* velc,
                             float dt, float inv_scale, int comp, nb_render_vertex* rv,
                             const float4* rcol, float rscale, const int32_t* hold,
                             int int_cap, int cell_cap, int* held) {
    wait_for_previous();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (hold && !tree_fits(hold, int_cap, cell_cap)) {   // the step is held: the state stays as it was
        if (i == 0) atomicAdd(held, 1);
        return;
    }
    const float4 a = acc[i];
    float4 v = vel[i], vc = velc[i], x = pos[i], xc = posc[i];
    if (comp) {
        kahan_add(v.x, vc.x, a.x * dt);
        kahan_add(v.y, vc.y, a.y * dt);
        kahan_add(v.z, vc.z, a.z * dt);
        kahan_add(x.x, xc.x, ((v.x - vc.x) * dt) * inv_scale);
        kahan_add(x.y, xc.y, ((v.y - vc.y) * dt) * inv_scale);
        kahan_add(x.z, xc.z, ((v.z - vc.z) * dt) * inv_scale);
        velc[i] = vc;
        posc[i] = xc;
    } else {
        v.x += a.x * dt; v.y += a.y * dt; v.z += a.z * dt;
        x.x += (v.x * dt) * inv_scale; x.y += (v.y * dt) * inv_scale; x.z += (v.z * dt) * inv_scale;
    }
    vel[i] = v;
    pos[i] = x;
    if (rv) write_vertex(rv, rcol, rscale, i, x);
}

namespace {

template <int LAW, int BLOCK, int IPT, bool COMP>
void launch_force_t(dim3 grid, cudaStream_t st, const float4* pos, int n_pad, int tps, int ntiles, int splits,
                    float S, float4* part, int* err, uint32_t polls, const unsigned* mmax, bool heavy) {
    if (heavy)
        k_direct_force<LAW, BLOCK, IPT, COMP, true><<<grid, BLOCK, 0, st>>>(pos, n_pad, tps, ntiles, splits, S, part,
                                                                           err, polls, mmax);
    else
        k_direct_force<LAW, BLOCK, IPT, COMP, false><<<grid, BLOCK, 0, st>>>(pos, n_pad, tps, ntiles, splits, S,
                                                                            part, err, polls, mmax);
}

template <int LAW, bool COMP>
bool launch_force_law(int block, int ipt, dim3 grid, cudaStream_t st, const float4* pos, int n_pad, int tps,
                      int ntiles, int splits, float S, float4* part, int* err, uint32_t polls,
                      const unsigned* mmax, bool heavy) {
#define NB_CASE(B, I)                                                                                    \
    if (block == B && ipt == I) {                                                                        \
        launch_force_t<LAW, B, I, COMP>(grid, st, pos, n_pad, tps, ntiles, splits, S, part, err, polls, mmax, heavy); \
        return true;                                                                                     \
    }
    NB_CASE(64, 1) NB_CASE(64, 2) NB_CASE(64, 4) NB_CASE(64, 8)
    NB_CASE(128, 1) NB_CASE(128, 2) NB_CASE(128, 4) NB_CASE(128, 8)
    NB_CASE(256, 1) NB_CASE(256, 2) NB_CASE(256, 4)
#undef NB_CASE
    return false;
}

}  // namespace

int direct_splits(const nb_sim* sim, const DirectTuning& t, size_t n_pad) {
    const int ntiles = (int)(n_pad / kTileJ);
    const int iblocks = (int)(n_pad / (size_t)(t.block * t.ipt));
    int splits = t.splits;
    if (splits <= 0) {
        const int target = std::max(1, sim->sm_count) * 256;  // many short units: dynamic balance
        splits = (target + iblocks - 1) / iblocks;
        // keep the partials (2 float4 per body per split) within 512 MB
        const size_t cap = (512ull << 20) / (n_pad * 2 * sizeof(float4));
        splits = (int)std::min<size_t>((size_t)splits, std::max<size_t>(1, cap));
    }
    splits = std::max(1, std::min(splits, ntiles));
    const int tps = (ntiles + splits - 1) / splits;
    return (ntiles + tps - 1) / tps;
}

static DirectTuning default_tuning(size_t n_pad) {
    DirectTuning t;
    t.block = 128;
    t.ipt = n_pad >= 16384 ? 2 : 1;
    return t;
}

static cudaError_t reserve_part(nb_sim* sim, size_t need) {
    if (need <= sim->part_cap) return cudaSuccess;
    dev_free(sim->part, sim->stream);
    sim->part = nullptr;
    sim->part_cap = 0;
    cudaError_t e = dev_alloc(&sim->part, need * sizeof(float4));
    if (e != cudaSuccess) return e;
    sim->part_cap = need;
    return cudaSuccess;
}

// k_direct_pairs over all rows in launches within cap entries of part, folded
// into the carry between launches.  The last launch's partials are left for the
// reduction (*last; *carry is null when it was the only one).  *made: the
// launches.  After a launch that failed nothing is queued behind it.
template <bool HEAVY, int FOLD>
static cudaError_t launch_pairs(int sm_count, int law, cudaStream_t st, const float4* pos, int n_pad, float S,
                                float4* part, size_t cap, bool all_rows, float4* carry_buf, int* err, uint32_t polls,
                                const unsigned* mmax, PairFold* last, const float4** carry, int* made) {
    const int rows = n_pad / kPairRow;
    *made = 0;
    *carry = nullptr;
    for (int r0 = 0; r0 < rows;) {
        const PairFold p = pair_plan(sm_count, n_pad, r0, cap, all_rows);
        const unsigned grid = (unsigned)pair_units(p, n_pad);
        if (law == NB_LAW_PLUMMER)
            k_direct_pairs<NB_LAW_PLUMMER, HEAVY, FOLD><<<grid, kPairThreads, 0, st>>>(pos, n_pad, r0, p.rows, p.per, S, part, err,
                                                                                 polls, mmax);
        else
            k_direct_pairs<NB_LAW_REFERENCE, HEAVY, FOLD><<<grid, kPairThreads, 0, st>>>(pos, n_pad, r0, p.rows, p.per, S, part, err,
                                                                                   polls, mmax);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        ++*made;
        *last = p;
        if (r0 + p.rows < rows) {
            k_pairs_carry<<<(unsigned)(n_pad / 32), 32 * kFoldWarps, 0, st>>>(part, p, n_pad, r0 == 0 ? 1 : 0, carry_buf, err);
            e = cudaGetLastError();
            if (e != cudaSuccess) return e;
            ++*made;
            *carry = carry_buf;
        }
        r0 += p.rows;
    }
    return cudaSuccess;
}

// Entries of partials a handle's k_direct_pairs launch may use (1 GiB): one
// launch up to about 360,000 bodies.
constexpr size_t kPairCap = ((size_t)1 << 30) / sizeof(float4);
// Padded bodies up to which single warps take the pairs (k_direct_rows), for a
// handle and in the allocation-free call, whose fixed array holds no more rows'
// partials.  A step of 8192 bodies takes 30 us by warps, of 10000 44 (k_direct_pairs
// 49), of 16384 95 (109), of 20480 146 (154), of 24000 199 (202): past that the
// row partials' own cost grows with the square of the bodies.
constexpr size_t kRowMax = 20480, kRowMaxNoAlloc = 8192;

// The units of k_direct_rows within cap entries of partials.  Short units spread
// over more warps, long ones leave fewer partials: a step with 1, 2 and 4 chunks a
// unit takes 5.8, 7.3 and 10.8 us at 1000 bodies, 9.2, 8.7 and 11.9 at 3000, 17.2, 16.3
// and 18.9 at 5000, 63, 56.4 and 56.9 at 12,000, 181, 147 and 140 at 20,000.
static size_t row_entries(const RowPlan& p, int n_pad) { return row_source_base(p, p.rows, n_pad); }

static RowPlan row_plan(int n, int n_pad, size_t cap) {
    RowPlan p;
    p.chunks = (n + kDirChunk - 1) / kDirChunk;
    p.rows = (n + kRowBodies - 1) / kRowBodies;
    p.per = p.chunks <= 64 ? 1 : p.chunks <= 256 ? 2 : 4;
    if (row_entries(p, n_pad) > cap) p.per = 4;
    return p;
}

static cudaError_t launch_rows(const RowPlan& p, int law, cudaStream_t st, const float4* pos, int n_pad, float S,
                        const unsigned* mmax, float4* part) {
    const unsigned grid = (unsigned)p.units_before(p.rows);
    return launch_after(law == NB_LAW_PLUMMER ? k_direct_rows<NB_LAW_PLUMMER> : k_direct_rows<NB_LAW_REFERENCE>, grid,
                        32, 0, st, pos, n_pad, p, S, mmax, part);
}

static cudaError_t force_pairs(nb_sim* sim, PairFold* last, const float4** carry) {
    const int n_pad = (int)sim->n_pad;
    size_t most = 0;
    cudaError_t e = cudaSuccess;
    // A handle that had to make do with less keeps to it until its state is
    // set up anew: no allocation is tried again on each step.
    const size_t cap = pair_reserve(sim->sm_count, n_pad, sim->pair_cap ? sim->pair_cap : kPairCap, &most, [&](size_t need) {
        e = reserve_part(sim, need);
        if (e == cudaErrorMemoryAllocation) cudaGetLastError();   // reported here or made good, not by the next launch
        return e != cudaErrorMemoryAllocation;
    });
    if (e != cudaSuccess) return e;
    if (cap != kPairCap) sim->pair_cap = cap;
    const float S = (float)sim->prm.softening2;
    auto go = sim->heavy ? launch_pairs<true, kFold> : launch_pairs<false, kFold>;
    int made = 0;
    e = go(sim->sm_count, sim->prm.law, sim->stream, sim->pos, n_pad, S, sim->part, cap, true, sim->part + most,
           sim->d_err, sim->wait_polls, sim->d_mmax, last, carry, &made);
    if (made > 1) sim->prof.launches += (uint64_t)(made - 1);   // the phase counts one
    return e;
}

cudaError_t direct_force_update(nb_sim* sim, float dt, bool update) {
    const bool comp = !(sim->prm.flags & NB_FLAG_NO_COMPENSATION);
    // Each pair once.  A handle whose launch was tuned, and uncompensated sums,
    // keep k_direct_force; so do small states whose waits were tuned
    // (k_direct_rows has none that could run out) and states beyond kPairMax.
    const bool small = sim->n_pad <= kRowMax;
    const bool once = comp && !sim->tune_set && sim->n_pad <= kPairMax && !(small && sim->wait_polls != kMaxPolls);
    const bool by_rows = once && small, pairs = once && !small;
    RowPlan rp{};
    int splits = 0;
    PairFold pf{};
    const float4* carry = nullptr;
    if (pairs) {
        PhaseScope ps(sim, 0);
        cudaError_t e = force_pairs(sim, &pf, &carry);
        if (e != cudaSuccess) return e;
    } else if (by_rows) {
        rp = row_plan((int)sim->n, (int)sim->n_pad, kPairCap);
        cudaError_t e = reserve_part(sim, row_entries(rp, (int)sim->n_pad));
        if (e == cudaErrorMemoryAllocation && rp.per < 4) {   // no room: longer units, fewer partials
            cudaGetLastError();
            rp.per = 4;
            e = reserve_part(sim, row_entries(rp, (int)sim->n_pad));
        }
        if (e != cudaSuccess) return e;
        PhaseScope ps(sim, 0);
        e = launch_rows(rp, sim->prm.law, sim->stream, sim->pos, (int)sim->n_pad, (float)sim->prm.softening2,
                        sim->heavy ? sim->d_mmax : nullptr, sim->part);
        if (e != cudaSuccess) return e;
    } else {
        DirectTuning t = sim->tune;
        if (!sim->tune_set) {
            t = default_tuning(sim->n_pad);
            t.splits = sim->tune.splits;
        }
        if (t.block <= 0 || t.ipt <= 0) t = default_tuning(sim->n_pad);
        // A tuning whose target block does not divide the padded size falls back.
        if (sim->n_pad % (size_t)(t.block * t.ipt) != 0) t = default_tuning(sim->n_pad);
        splits = direct_splits(sim, t, sim->n_pad);
        cudaError_t e = reserve_part(sim, (size_t)splits * 2 * sim->n_pad);
        if (e != cudaSuccess) return e;
        const int ntiles = (int)(sim->n_pad / kTileJ);
        const int tps = (ntiles + splits - 1) / splits;
        dim3 grid((unsigned)(sim->n_pad / (size_t)(t.block * t.ipt)), (unsigned)splits);
        const float S = (float)sim->prm.softening2;
        bool ok;
        PhaseScope ps(sim, 0);
#define NB_FORCE(L, C)                                                                                               \
    ok = launch_force_law<L, C>(t.block, t.ipt, grid, sim->stream, sim->pos, (int)sim->n_pad, tps, ntiles, splits, S, \
                                sim->part, sim->d_err, sim->wait_polls, sim->d_mmax, sim->heavy)
        if (sim->prm.law == NB_LAW_PLUMMER) { if (comp) NB_FORCE(NB_LAW_PLUMMER, true); else NB_FORCE(NB_LAW_PLUMMER, false); }
        else { if (comp) NB_FORCE(NB_LAW_REFERENCE, true); else NB_FORCE(NB_LAW_REFERENCE, false); }
#undef NB_FORCE
        if (!ok) return cudaErrorInvalidConfiguration;
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    const int n = (int)sim->n;
    const UpdateArgs ua{(float)sim->prm.G, dt, (float)(1.0 / sim->prm.pos_scale), update ? 1 : 0, comp ? 1 : 0,
                        sim->finit_pending ? sim->finit : nullptr, sim->acc, sim->pos, sim->posc, sim->vel, sim->velc,
                        update ? sim->render : nullptr, sim->rcolour, sim->rscale};
    sim->finit_pending = false;
    const double nn = (double)sim->n;
    sim->inter_last = (uint64_t)(nn * (nn - 1.0));
    PhaseScope ps(sim, 1);
    static_assert(kPad % (256 / kFoldLanes) == 0 && kPad % 32 == 0, "the fold's blocks cover whole padded bodies");
    if (pairs)
        k_direct_pairs_update<<<(unsigned)((n + 31) / 32), 32 * kFoldWarps, 0, sim->stream>>>(
            sim->part, pf, carry, n, (int)sim->n_pad, ua, sim->d_err);
    else if (by_rows)
        return launch_after(k_direct_rows_update, (unsigned)((n + 31) / 32), 32 * kFoldWarps, 0, sim->stream,
                            sim->part, rp, n, (int)sim->n_pad, ua, sim->d_err);
    else
        k_direct_reduce_update<<<(unsigned)(sim->n_pad * kFoldLanes / 256), 256, 0, sim->stream>>>(
            sim->part, splits, n, (int)sim->n_pad, ua, sim->d_err);
    return cudaGetLastError();
}

cudaError_t kick_drift(nb_sim* sim, float dt, const int32_t* hold, int int_cap, int cell_cap, int* held) {
    const int n = (int)sim->n;
    const bool comp = !(sim->prm.flags & NB_FLAG_NO_COMPENSATION);
    PhaseScope ps(sim, 7);
    return launch_after(k_kick_drift, (n + 255) / 256, 256, 0, sim->stream, sim->acc, n, sim->pos, sim->posc,
                        sim->vel, sim->velc, dt, (float)(1.0 / sim->prm.pos_scale), comp ? 1 : 0, sim->render,
                        sim->rcolour, sim->rscale, hold, int_cap, cell_cap, held);
}

}  // namespace nb

// ---------------------------------------------------------------------------
// Allocation-free direct-sum accelerations.
//
// For callers that must not allocate device memory while they step: a render
// loop that stays inside a fixed device-memory budget, a host that hands in
// buffers owned by its own allocator, or a thread that must not block (every
// cudaFree synchronises the whole device).  The caller passes device input
// and output buffers; the working memory of the kernels is a file-scope
// __device__ array of fixed size that every GPU loading this library holds
// until the process exits.  It has no counterpart in the reference.
// ---------------------------------------------------------------------------
#include <mutex>

namespace nb {

// padded copy of the input + 16 entries of partials a body at the most bodies
constexpr size_t kNoAllocScratch = (size_t)NB_NOALLOC_MAX_BODIES * 17;
static_assert((kRowMaxNoAlloc / (4 * kDirChunk) + kRowMaxNoAlloc / kRowBodies / 2 + 1) * kRowMaxNoAlloc <= kNoAllocScratch,
              "the array holds the rows' partials at four chunks a unit");
static __device__ __align__(256) float4 g_noalloc_scratch[kNoAllocScratch];   // 17.8 MB
static __device__ int g_noalloc_err;
// float bits of the call's largest |mass| (the force law's self-pair guard);
// zero between calls: the reduce kernel clears it after the force kernel read it
static __device__ unsigned g_noalloc_mmax;

// Copies n bodies into the scratch and zero-fills the padding (zero-mass
// bodies at the origin contribute exactly nothing); clears the error word and
// records the largest |mass|.
__global__ void k_noalloc_stage(const float4* __restrict__ in, int n, int n_pad, float4* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) g_noalloc_err = 0;
    if (i < n_pad) {
        const float4 p = i < n ? in[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        out[i] = p;
        if (i < n) atomicMax(&g_noalloc_mmax, __float_as_uint(fabsf(p.w)));
    }
}

// Folds the partials like k_direct_reduce_update; a force kernel whose bounded
// wait ran out poisons the output with NaN, since nothing is read back.
__global__ void __launch_bounds__(32 * kFoldWarps) k_noalloc_reduce(const float4* __restrict__ part, PairFold pf,
                                                                    const float4* __restrict__ carry, int n, int n_pad,
                                                                    float G, float4* __restrict__ acc) {
    __shared__ float sums[kFoldWarps][6][32];
    const int i = blockIdx.x * 32 + (threadIdx.x & 31), j = threadIdx.x >> 5;
    const HiLo3 f = fold_pairs(part, pf, n_pad, i, j, sums);
    if (i >= n || j != 0) return;
    const float3 s = with_carry(f, carry, n_pad, i);
    float4 a = make_float4(G * s.x, G * s.y, G * s.z, 0.f);
    if (g_noalloc_err != 0) a = make_float4(NAN, NAN, NAN, NAN);
    acc[i] = a;
    if (i == 0) g_noalloc_mmax = 0u;
}

// The same for k_direct_rows (which has no wait to run out).
__global__ void __launch_bounds__(32 * kFoldWarps) k_noalloc_rows(const float4* part, RowPlan plan, int n, int n_pad,
                                                                float G, float4* acc) {
    __shared__ float sums[kFoldWarps][6][32];
    const int i = blockIdx.x * 32 + (threadIdx.x & 31), j = threadIdx.x >> 5;
    const float3 s = fold_rows(part, plan, n_pad, i, j, sums);
    if (i >= n || j != 0) return;
    acc[i] = make_float4(G * s.x, G * s.y, G * s.z, 0.f);
    if (i == 0) g_noalloc_mmax = 0u;
}

namespace {
std::mutex g_noalloc_mu;
float4* g_noalloc_ptr[256] = {};   // device address of the scratch, per device ordinal
int* g_noalloc_err_ptr[256] = {};
unsigned* g_noalloc_mmax_ptr[256] = {};
}  // namespace

}  // namespace nb

extern "C" int nb_direct_accel_noalloc(const float* pos_mass4, size_t n, float* accel4, double G, double softening2,
                                       int law, void* stream) {
    using namespace nb;
    if (!pos_mass4 || !accel4 || n == 0) return NB_EINVAL;
    if (n > (size_t)NB_NOALLOC_MAX_BODIES) return NB_EINVAL;
    if (law != NB_LAW_REFERENCE && law != NB_LAW_PLUMMER) return NB_EINVAL;
    if (!std::isfinite(G) || !std::isfinite(softening2) || softening2 < 0 ||
        (law == NB_LAW_PLUMMER && softening2 <= 0))
        return NB_EINVAL;
    if ((reinterpret_cast<uintptr_t>(pos_mass4) | reinterpret_cast<uintptr_t>(accel4)) & 15u) return NB_EINVAL;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) { cudaGetLastError(); return NB_ECUDA; }
    float4* scratch = nullptr;
    int* err = nullptr;
    unsigned* mmax = nullptr;
    {
        // Set-up on the first call on each device, with that device current.
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        if (!g_noalloc_ptr[dev]) {
            void* p = nullptr;
            void* q = nullptr;
            void* r = nullptr;
            if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess ||
                cudaGetSymbolAddress(&q, g_noalloc_err) != cudaSuccess ||
                cudaGetSymbolAddress(&r, g_noalloc_mmax) != cudaSuccess || !p || !q || !r) {
                cudaGetLastError();
                return NB_ECUDA;
            }
            g_noalloc_ptr[dev] = static_cast<float4*>(p);
            g_noalloc_err_ptr[dev] = static_cast<int*>(q);
            g_noalloc_mmax_ptr[dev] = static_cast<unsigned*>(r);
        }
        scratch = g_noalloc_ptr[dev];
        err = g_noalloc_err_ptr[dev];
        mmax = g_noalloc_mmax_ptr[dev];
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t n_pad = pad_up(n, kPad);
    float4* pos = scratch;
    float4* part = scratch + n_pad;
    const float S = (float)softening2;
    k_noalloc_stage<<<(unsigned)((n_pad + 255) / 256), 256, 0, st>>>(reinterpret_cast<const float4*>(pos_mass4),
                                                                    (int)n, (int)n_pad, pos);
    float4* acc = reinterpret_cast<float4*>(accel4);
    if (n_pad <= kRowMaxNoAlloc) {
        const RowPlan rp = row_plan((int)n, (int)n_pad, kNoAllocScratch - n_pad);
        if (launch_rows(rp, law, st, pos, (int)n_pad, S, mmax, part) != cudaSuccess) return NB_ECUDA;
        k_noalloc_rows<<<(unsigned)((n + 31) / 32), 32 * kFoldWarps, 0, st>>>(part, rp, (int)n, (int)n_pad, (float)G, acc);
    } else {
        PairFold pf{};
        const float4* carry = nullptr;
        // Each pair once, as for a handle, in as many launches as the fixed array
        // asks for (six at 65,536 bodies; two entries a body hold their running
        // sums).  Folding targets every 16 sources instead of 32 costs 4% and
        // keeps the error at or below that of the one-direction kernel, whose
        // fold here rounded less than the handle's did.  GB300: 50,001 bodies
        // 1257 -> 946 us, 65,536 2004 -> 1530, 20,000 260 -> 191, 10,000 86 -> 54.
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
            cudaGetLastError();
            return NB_ECUDA;
        }
        const size_t cap = kNoAllocScratch - 3 * n_pad;
        int made = 0;
        if (launch_pairs<true, kFold / 2>(sms, law, st, pos, (int)n_pad, S, part, cap, false, part + cap, err, kMaxPolls, mmax,
                                          &pf, &carry, &made) != cudaSuccess)
            return NB_ECUDA;
        k_noalloc_reduce<<<(unsigned)((n + 31) / 32), 32 * kFoldWarps, 0, st>>>(part, pf, carry, (int)n, (int)n_pad, (float)G,
                                                                                acc);
    }
    if (cudaGetLastError() != cudaSuccess) return NB_ECUDA;
    return NB_OK;
}
