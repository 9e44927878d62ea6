// nb_tree.cu -- Barnes-Hut octree build on the GPU: K2 keys, K3 radix sort,
// K4 topology, K5 bottom-up mass and centre of mass.
//
// Replaces the serial pointer octree of BarnesHut::Update
// (src/Sim/BarnesHut.cpp:44-56) and Octree::Split/Add/CalculateMass
// (src/Sim/Octree.cpp:16-105) with the same tree, built in parallel:
//
//  * K2: a body's key is the octant path Octree::Add takes from the root,
//    3 bits per level, octant = x + 2y + 4z (src/Sim/Octree.cpp:25-41).  The
//    child bounds are replayed in float exactly as Split computes them
//    (cur += size, BottomRight = cur + size, Size = BottomRight.x - TopLeft.x),
//    with the half-open containment of BoundingCube::Contains
//    (src/Sim/Octree.hpp:18-22).  A body outside the root cube gets key ~0:
//    the reference drops it from the tree but counts it in the root.
//  * K3: stable LSD radix sort of (key, body) pairs, 8 passes of 8 bits, one
//    launch per pass: the digit histograms of all passes come with the keys,
//    and each pass ranks, finds its tile's offsets by decoupled look-back and
//    scatters in one kernel (digits are ranked by warp ballots); small states
//    are sorted whole by one block.
//    Passes whose digit is the same for every key are skipped on the device.
//  * K4: the reference tree splits a node when a second body arrives and
//    creates all 8 children, so its internal nodes are exactly the key
//    prefixes shared by at least two bodies (and the root whenever it holds
//    two bodies, dropped ones included).  With sorted keys, delta(s) = the
//    number of leading octants bodies s and s+1 share; position s starts the
//    internal nodes of levels delta(s-1)+1 .. min(delta(s), D-1) and one
//    leaf.  Internal nodes are numbered by (first body, level) through a
//    prefix sum; a node whose parent starts at an earlier body finds it in a
//    hash table keyed by (1 << 3 level) | prefix.  Each internal node stores
//    only its non-empty children, as consecutive cells in octant order
//    (empty children hold no mass and contribute exactly zero force).
//  * Depth cap D (max_depth, 21 = 63-bit keys): bodies sharing all D octants
//    form one leaf (a bucket).  A bucket's mass and centre of mass sum its
//    bodies in ascending body index (stable sort order).
//  * K5: CalculateMass in the same arithmetic: TotalMass is a double sum of
//    the children in octant order, CentreOfMass += child COM * float(child
//    mass) in float, then scaled by 1.f / float(TotalMass).  Nodes are
//    finished bottom-up: the last child to arrive finishes its parent.
#include "nb_common.cuh"
#include "nb_internal.hpp"
#include "nb_scan.cuh"
#include "nb_lookback.cuh"
#include "nb_morton.cuh"
#include "nb_cellrec.cuh"
#include "nb_hilbert.cuh"
#include "nb_tree_nodes.hpp"
#include <algorithm>
#include <cmath>
#include <cstring>

namespace nb {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;   // 4096 keys per tile
// a radix pass ranks a tile with more threads and fewer keys each (more warps
// in flight to hide the loads); at most 64 registers, two blocks per SM
constexpr int kPassThreads = 512;
constexpr int kPassWarps = kPassThreads / 32;
constexpr int kPassItems = kSortTile / kPassThreads;
constexpr int kPasses = 8;
constexpr int kEmitBlock = 256;

enum : int { KIND_SINGLE = 1, KIND_BUCKET = 2, KIND_INTERNAL = 3 };

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// ---------------------------------------------------------------- K2 keys --
// The octant path of body p (Octree::Add's descent) and its length; gap: the
// path met a gap between float child bounds and was cut short.  A body that a
// cell holds is never below the cell's lower bound, so an axis takes the upper
// half when p >= middle and only there can it miss (p beyond middle + size, the
// float sum the upper child ends at).  No branch a level: the three axes of 32
// bodies go eight ways.
__device__ __forceinline__ uint64_t body_key(const float4 p, float half, int D, bool& inside, bool& gap, int& d) {
    float lo0 = -half, lo1 = -half, lo2 = -half;
    const float hi = half;
    inside = p.x >= lo0 && p.y >= lo1 && p.z >= lo2 && p.x < hi && p.y < hi && p.z < hi;
    gap = false;
    d = 0;
    if (!inside) return ~0ull;
    uint64_t key = 0;
    float size = __fsub_rn(hi, lo0);
    for (int l = 0; l < D; ++l) {
        const float s = __fmul_rn(size, 0.5f);   // Size / 2: exact halving, the same value as a division
        const float m0 = __fadd_rn(lo0, s), m1 = __fadd_rn(lo1, s), m2 = __fadd_rn(lo2, s);
        const float t0 = __fadd_rn(m0, s), t1 = __fadd_rn(m1, s), t2 = __fadd_rn(m2, s);
        const bool u0 = p.x >= m0, u1 = p.y >= m1, u2 = p.z >= m2;
        if ((u0 && !(p.x < t0)) || (u1 && !(p.y < t1)) || (u2 && !(p.z < t2))) break;
        size = u0 ? __fsub_rn(t0, m0) : __fsub_rn(m0, lo0);   // the child's extent along x
        lo0 = u0 ? m0 : lo0;
        lo1 = u1 ? m1 : lo1;
        lo2 = u2 ? m2 : lo2;
        key = (key << 3) | (uint64_t)((u0 ? 1u : 0u) | (u1 ? 2u : 0u) | (u2 ? 4u : 0u));
        ++d;
    }
    if (d < D) {   // a gap between float child bounds: left-align the path
        key <<= 3 * (D - d);
        gap = true;
    }
    return key;
}

// Keys per thread of the keys kernels.  A key is a chain of ~21 dependent float
// steps, so a block of few keys a thread hides it behind other blocks: a whole
// 4096-key tile a block left 25 blocks at 100,000 bodies and one at 4,000
// (64 us either way).  More keys a thread only pays once every SM holds its
// eight blocks, by fewer histogram flushes.
inline int keys_per_thread(size_t nk, int sm_count) {
    int items = 1;
    while (items < 4 && nk / (size_t)(kSortThreads * items * 2) >= (size_t)(8 * sm_count)) items *= 2;
    return items;
}

// Zeroes the look-back status words of every radix pass and of the positions
// scan, spread over the grid.
__device__ __forceinline__ void zero_tile_status(unsigned long long* sort_status, int ntiles,
                                                 unsigned long long* pos_status, int blocks) {
    const int words = kPasses * ntiles * 256;
    for (int i = blockIdx.x * kSortThreads + threadIdx.x; i < words; i += blocks * kSortThreads) sort_status[i] = 0ull;
    for (int i = blockIdx.x * kSortThreads + threadIdx.x; i < ntiles; i += blocks * kSortThreads) pos_status[i] = 0ull;
}

// Radix passes that the top bits make redundant.  Keys are grouped by their
// top 4 bits (the root octant, and ~0 for bodies outside the root or tile
// padding), which the top pass sorts.  A lower pass whose digit is the same
// for every key of each group changes nothing in the final order: the top pass
// orders the groups, and within a group that digit is constant, so the order
// within the group is that of the passes below it.  Such a pass is skipped.
// For a galaxy at the centre of the reference's +-4000 cube, the bits of
// levels 2-7 are fixed within each root octant: two of the eight passes go.
// The group bits are recorded as two ORs per group, of the keys and of their
// complements (both start at zero with the counters): a bit varies within
// group g where both have it.
constexpr int kKeyGroups = 16;
__device__ __forceinline__ unsigned long long* group_bits(uint32_t* ghist) {
    return reinterpret_cast<unsigned long long*>(ghist + kPasses * 256);
}

// Counts a warp's keys into the digit histograms and the group bits in shared
// memory.  A digit that the whole warp shares (the upper levels of a galaxy
// that fills a small part of the root cube) is added once for the warp: 32
// atomics on one word would be done one after the other.
__device__ __forceinline__ void count_key(uint64_t key, uint32_t (*h)[256], unsigned long long* sh) {
    const uint32_t full = 0xffffffffu;
    const uint32_t lo = (uint32_t)key, hi = (uint32_t)(key >> 32);
    const uint32_t olo = __reduce_or_sync(full, lo), ohi = __reduce_or_sync(full, hi);
    const uint32_t zlo = __reduce_or_sync(full, ~lo), zhi = __reduce_or_sync(full, ~hi);
    const uint64_t o = ((uint64_t)ohi << 32) | olo, z = ((uint64_t)zhi << 32) | zlo;
    const uint64_t varies = o & z;   // bits that differ within the warp
    const bool first = (threadIdx.x & 31) == 0;
#pragma unroll
    for (int p = 0; p < kPasses; ++p) {
        const uint32_t d = (uint32_t)(key >> (8 * p)) & 255u;
        if (((varies >> (8 * p)) & 255ull) == 0ull) {
            if (first) atomicAdd(&h[p][d], 32u);
        } else {
            atomicAdd(&h[p][d], 1u);
        }
    }
    const uint32_t g = (uint32_t)(key >> 60);
    if ((varies >> 60) == 0ull) {
        if (first) {
            atomicOr(&sh[g], (unsigned long long)o);
            atomicOr(&sh[kKeyGroups + g], (unsigned long long)z);
        }
    } else {
        atomicOr(&sh[g], (unsigned long long)key);
        atomicOr(&sh[kKeyGroups + g], (unsigned long long)~key);
    }
}

// Adds a block's digit histograms of every pass into ghist (bins that are
// zero in this block cost nothing), and its group bits after them.
__device__ __forceinline__ void flush_hist(uint32_t (*h)[256], const unsigned long long* sh_groups, uint32_t* ghist) {
    __syncthreads();
    for (int i = threadIdx.x; i < kPasses * 256; i += kSortThreads) {
        const uint32_t v = (&h[0][0])[i];
        if (v) atomicAdd(&ghist[i], v);
    }
    if (threadIdx.x < 2 * kKeyGroups && sh_groups[threadIdx.x])
        atomicOr(&group_bits(ghist)[threadIdx.x], sh_groups[threadIdx.x]);
}

// K2 + the radix sort's global histograms: kSortThreads * items keys a block
// (key ~0 past n); counts bodies inside the root and paths cut by gaps.  With
// curve, the keys are the paths in Hilbert order (nb_hilbert.cuh).
// Bound by the descent's arithmetic (~21 levels a key) once there are enough
// blocks; before, by one long chain a thread and, at 1M, by 32,768 atomics on
// the body count.  GB300, events: 4,000 bodies 62 -> 10 us, 100,003 64 -> 12 us,
// 1,048,576 74 -> 41 us.
__global__ void __launch_bounds__(kSortThreads) k_keys_hist(const float4* __restrict__ pos, int n, float half, int D,
                                                            uint64_t* __restrict__ keys, int32_t* __restrict__ vals,
                                                            int32_t* __restrict__ depth,
                                                            int32_t* __restrict__ counters, uint32_t* __restrict__ ghist,
                                                            unsigned long long* __restrict__ sort_status, int ntiles,
                                                            unsigned long long* __restrict__ pos_status, int items,
                                                            bool curve) {
    __shared__ uint32_t table[2 * kHilbertStates];
    __shared__ uint32_t h[kPasses][256];
    __shared__ unsigned long long sh_groups[2 * kKeyGroups];
    __shared__ int sh_in, sh_gaps;   // one global atomic a block: one a warp queued 32,768 on one word at 1M
    for (int i = threadIdx.x; i < kPasses * 256; i += kSortThreads) (&h[0][0])[i] = 0;
    if (threadIdx.x < 2 * kKeyGroups) sh_groups[threadIdx.x] = 0ull;
    if (threadIdx.x == 0) sh_in = sh_gaps = 0;
    load_hilbert(table, false);
    zero_tile_status(sort_status, ntiles, pos_status, gridDim.x);
    __syncthreads();
    for (int it = 0; it < items; ++it) {
        const int i = (blockIdx.x * items + it) * kSortThreads + threadIdx.x;
        vals[i] = i;
        bool inside = false, gap = false;
        uint64_t key = ~0ull;
        if (i < n) {
            int d;
            key = body_key(pos[i], half, D, inside, gap, d);
            depth[i] = d;
            if (curve && inside) key = hilbert_map_cut(key, d, D, table);
        }
        keys[i] = key;
        count_key(key, h, sh_groups);
        const uint32_t in_b = __ballot_sync(0xffffffffu, inside);
        const uint32_t gap_b = __ballot_sync(0xffffffffu, gap);
        if ((threadIdx.x & 31) == 0) {
            if (in_b) atomicAdd(&sh_in, __popc(in_b));
            if (gap_b) atomicAdd(&sh_gaps, __popc(gap_b));
        }
    }
    flush_hist(h, sh_groups, ghist);
    if (threadIdx.x == 0) {
        if (sh_in) atomicAdd(&counters[TC_NIN], sh_in);
        if (sh_gaps) atomicAdd(&counters[TC_GAPS], sh_gaps);
    }
}

// ------------------------------------------------------------ K3 radix sort --
// plan[p] = 1 when pass p is skipped: every key has the same digit, or (below
// the top pass) every key of each top group has (count_key); plan[8+p] =
// buffer the pass reads; plan[16] = buffer holding the result.  dig_off[p][d] = keys
// with a smaller digit than d in pass p (where digit d's keys start).
// One warp per pass, eight digits a lane: 8.3 -> 4 us against eight block scans
// one after the other (ncu).
static_assert(kPasses * 32 == 256, "one warp per pass");
__global__ void __launch_bounds__(256) k_sort_plan(const uint32_t* ghist, int nk,
                                                   int32_t* plan, int32_t* dig_off) {
    wait_for_previous();
    __shared__ int triv[kPasses];
    const int p = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint4* bins = reinterpret_cast<const uint4*>(ghist + p * 256) + 2 * lane;
    const uint4 a = bins[0], b = bins[1];
    // bits that vary within some top group
    const unsigned long long* gb = group_bits(const_cast<uint32_t*>(ghist));
    const unsigned long long v = lane < kKeyGroups ? gb[lane] & gb[kKeyGroups + lane] : 0ull;
    const uint32_t vlo = __reduce_or_sync(0xffffffffu, (uint32_t)v);
    const uint32_t vhi = __reduce_or_sync(0xffffffffu, (uint32_t)(v >> 32));
    const unsigned long long var = ((unsigned long long)vhi << 32) | vlo;
    const int c[8] = {(int)a.x, (int)a.y, (int)a.z, (int)a.w, (int)b.x, (int)b.y, (int)b.z, (int)b.w};
    int sum = 0;
    bool all = false;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        sum += c[k];
        all |= c[k] == nk;
    }
    int run = warp_incl_scan(sum) - sum;
    int4 o[2];
    int* of = reinterpret_cast<int*>(o);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        of[k] = run;
        run += c[k];
    }
    int4* out = reinterpret_cast<int4*>(dig_off + p * 256) + 2 * lane;
    out[0] = o[0];
    out[1] = o[1];
    const bool one = __any_sync(0xffffffffu, all);
    if (lane == 0) triv[p] = one || (p < kPasses - 1 && ((var >> (8 * p)) & 255ull) == 0ull);
    __syncthreads();
    if (threadIdx.x == 0) {
        int cur = 0;
        for (int q = 0; q < kPasses; ++q) {
            plan[q] = triv[q];
            plan[8 + q] = cur;
            if (!triv[q]) cur ^= 1;
        }
        plan[16] = cur;
    }
}

// The lanes of the warp that hold the same 8-bit digit: eight ballots.  (One
// __match_any_sync goes through the warp's distinct values one by one: a pass
// over one tile of random digits took 13 us with it, 6.5 us over equal ones.)
__device__ __forceinline__ uint32_t same_digit(uint32_t d) {
    uint32_t peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool set = (d >> b) & 1u;
        const uint32_t m = __ballot_sync(0xffffffffu, set);
        peers &= set ? m : ~m;
    }
    return peers;
}

// Stable ranks of a warp's keys (in the order it, lane) among its keys of the
// same digit, each given to put(item, rank); hist (zero before) receives the warp's digit counts.
template <int ITEMS, class Put>
__device__ __forceinline__ void rank_keys(const uint64_t (&k)[ITEMS], int shift, uint16_t* hist, Put put) {
    const uint32_t lt = lanemask_lt();
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        const uint32_t d = (uint32_t)(k[it] >> shift) & 255u;
        const uint32_t peers = same_digit(d);
        const uint32_t b = hist[d];
        put(it, b + __popc(peers & lt));
        __syncwarp();
        if (lane == 31 - __clz(peers)) hist[d] = (uint16_t)(b + __popc(peers));
        __syncwarp();
    }
}

// Turns the warps' digit counts into each warp's first place among the block's
// keys of the digit; returns, in threads 0..255, the block's keys of digit
// threadIdx.x.  Every thread of the block calls it: a warp takes 32 digits of
// WARPS / SHARE rows (no bank conflicts), SHARE warps a digit.
template <int THREADS>
__device__ __forceinline__ uint32_t warp_places(uint16_t (*whist)[256], uint32_t (*count)[256]) {
    constexpr int WARPS = THREADS / 32, SHARE = THREADS / 256, EACH = WARPS / SHARE;
    const int d = threadIdx.x & 255, q = threadIdx.x >> 8;
    uint32_t c[EACH], sum = 0;
#pragma unroll
    for (int w = 0; w < EACH; ++w) {
        c[w] = whist[q * EACH + w][d];
        sum += c[w];
    }
    count[q][d] = sum;
    __syncthreads();
    uint32_t run = 0, all = 0;
#pragma unroll
    for (int o = 0; o < SHARE; ++o) {
        const uint32_t t = count[o][d];
        all += t;
        if (o < q) run += t;
    }
#pragma unroll
    for (int w = 0; w < EACH; ++w) {
        whist[q * EACH + w][d] = (uint16_t)run;
        run += c[w];
    }
    return threadIdx.x < 256 ? all : 0u;
}

// One pass of the stable LSD sort in one launch (the one-sweep scheme,
// Adinets and Merrill 2022): a tile ranks its keys by the pass's digit
// (warps in order: stable), publishes its digit counts and finds where earlier
// tiles put theirs by decoupled look-back.  The keys, then the indices, go
// through shared memory in the tile's order, so that neighbouring threads
// write neighbouring words: the sort of 2^20 keys took 141 us with match_any
// and a direct scatter, takes 98 (eight passes at 24 bytes a key: 28 us of
// copying; the rest is the latency of load, rank, look-back and scatter in
// about one wave of tiles).
__global__ void __launch_bounds__(kPassThreads, 2) k_sort_pass(uint64_t* k0, uint64_t* k1,
                                                            int32_t* v0, int32_t* v1,
                                                            int ntiles, const int32_t* plan, int pass,
                                                            const int32_t* dig_off,
                                                            unsigned long long* status,
                                                            int* tile_ctr, int* err) {
    wait_for_previous();
    if (plan[pass]) return;
    const int src = plan[8 + pass];
    const uint64_t* ks = src ? k1 : k0;
    uint64_t* kd = src ? k0 : k1;
    const int32_t* vs = src ? v1 : v0;
    int32_t* vd = src ? v0 : v1;
    __shared__ __align__(16) uint64_t stage[kSortTile];
    __shared__ __align__(16) uint16_t whist[kPassWarps][256];
    __shared__ uint32_t count[kPassThreads / 256][256];
    __shared__ int32_t start[256], shift_to[256];   // the tile's first key of a digit; its place less that
    __shared__ int sh_warp[33], sh_tile;
    const int tile = lb_tile_index(tile_ctr, &sh_tile);
    if (tile >= ntiles) return;   // cannot happen with one block per tile; kept as a guard
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int shift = 8 * pass;
    const int base = tile * kSortTile + warp * (32 * kPassItems) + lane;
    uint64_t k[kPassItems];
    int32_t v[kPassItems];
    uint32_t r[kPassItems];
#pragma unroll
    for (int it = 0; it < kPassItems; ++it) {
        k[it] = ks[base + it * 32];
        v[it] = vs[base + it * 32];
    }
    for (int i = threadIdx.x; i < kPassWarps * 256 / 8; i += kPassThreads)
        reinterpret_cast<uint4*>(&whist[0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    rank_keys<kPassItems>(k, shift, whist[warp], [&](int it, uint32_t rank) { r[it] = rank; });
    __syncthreads();
    const uint32_t mine = warp_places<kPassThreads>(whist, count);
    uint32_t excl = 0;
    if (threadIdx.x < 256) {   // one thread per digit
        const int d = threadIdx.x;
        unsigned long long* st = status + (size_t)tile * 256 + d;
        if (tile == 0) {
            lb_publish(st, 2u, mine);
        } else {
            lb_publish(st, 1u, mine);
            excl = lb_exclusive(status + d, tile, 256, err);
            lb_publish(st, 2u, excl + mine);
        }
    }
    int total;
    const int first = block_excl_scan((int)mine, sh_warp, &total);   // threads past the digits add nothing
    if (threadIdx.x < 256) {
        start[threadIdx.x] = first;
        shift_to[threadIdx.x] = dig_off[pass * 256 + threadIdx.x] + (int)excl - first;
    }
    __syncthreads();
    int place[kPassItems];
#pragma unroll
    for (int it = 0; it < kPassItems; ++it) {
        const uint32_t d = (uint32_t)(k[it] >> shift) & 255u;
        place[it] = start[d] + (int)whist[warp][d] + (int)r[it];
        stage[place[it]] = k[it];
    }
    __syncthreads();
    int dst[kPassItems];
#pragma unroll
    for (int it = 0; it < kPassItems; ++it) {
        const int j = it * kPassThreads + threadIdx.x;
        const uint64_t key = stage[j];
        dst[it] = shift_to[(uint32_t)(key >> shift) & 255u] + j;
        kd[dst[it]] = key;
    }
    __syncthreads();
    int32_t* vstage = reinterpret_cast<int32_t*>(stage);
#pragma unroll
    for (int it = 0; it < kPassItems; ++it) vstage[place[it]] = v[it];
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kPassItems; ++it) vd[dst[it]] = vstage[it * kPassThreads + threadIdx.x];
}

// The whole sort of one tile's keys in one block: every pass ranks the keys in
// registers and reorders them in shared memory, where the plan and one launch per
// pass cost 40 to 50 us however few the keys: 27 to 36 us for 4000 keys.  (Two
// tiles so took 46 us against 44, with four keys more a thread to keep.)  The
// keys end in buffer 0.
constexpr int kOneThreads = 1024, kOneWarps = kOneThreads / 32, kOneItems = kSortTile / kOneThreads;
constexpr size_t kOneBytes = (size_t)kSortTile * 10 + (size_t)kOneWarps * 256 * 2;   // keys, indices, histograms
__global__ void __launch_bounds__(kOneThreads) k_sort_block(uint64_t* keys, int32_t* vals, const uint32_t* ghist,
                                                            int32_t* plan) {
    wait_for_previous();
    constexpr int N = kSortTile, ITEMS = kOneItems;
    extern __shared__ __align__(16) unsigned char sm[];
    uint64_t* sk = reinterpret_cast<uint64_t*>(sm);
    uint16_t* sv = reinterpret_cast<uint16_t*>(sk + N);
    uint16_t (*whist)[256] = reinterpret_cast<uint16_t (*)[256]>(sv + N);
    __shared__ uint32_t count[kOneThreads / 256][256];
    __shared__ int32_t start[256];
    __shared__ int sh_warp[33], triv[kPasses];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int base = warp * (32 * ITEMS) + lane;
    if (warp < kPasses) {   // the passes to skip, as in k_sort_plan
        const uint4* bins = reinterpret_cast<const uint4*>(ghist + warp * 256) + 2 * lane;
        const uint4 a = bins[0], b = bins[1];
        const unsigned long long* gb = group_bits(const_cast<uint32_t*>(ghist));
        const unsigned long long v = lane < kKeyGroups ? gb[lane] & gb[kKeyGroups + lane] : 0ull;
        const unsigned long long var = ((unsigned long long)__reduce_or_sync(0xffffffffu, (uint32_t)(v >> 32)) << 32) |
                                       __reduce_or_sync(0xffffffffu, (uint32_t)v);
        const uint32_t n = (uint32_t)N;
        const bool all = a.x == n || a.y == n || a.z == n || a.w == n || b.x == n || b.y == n || b.z == n || b.w == n;
        const bool one = __any_sync(0xffffffffu, all);
        if (lane == 0) triv[warp] = one || (warp < kPasses - 1 && ((var >> (8 * warp)) & 255ull) == 0ull);
    }
    uint64_t k[ITEMS];
    uint32_t rv[ITEMS];   // a key's index (low half: below kSortTile) and its rank
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        k[it] = keys[base + it * 32];
        rv[it] = (uint32_t)(base + it * 32);   // the keys come in input order
    }
    __syncthreads();
    for (int pass = 0; pass < kPasses; ++pass) {
        if (triv[pass]) continue;   // block-uniform
        const int shift = 8 * pass;
        for (int i = threadIdx.x; i < kOneWarps * 256 / 8; i += kOneThreads)
            reinterpret_cast<uint4*>(&whist[0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        rank_keys<ITEMS>(k, shift, whist[warp], [&](int it, uint32_t r) { rv[it] |= r << 16; });
        __syncthreads();
        const uint32_t mine = warp_places<kOneThreads>(whist, count);
        int total;
        const int first = block_excl_scan((int)mine, sh_warp, &total);
        if (threadIdx.x < 256) start[threadIdx.x] = first;
        __syncthreads();
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
            const uint32_t d = (uint32_t)(k[it] >> shift) & 255u;
            const int p = start[d] + (int)whist[warp][d] + (int)(rv[it] >> 16);
            sk[p] = k[it];
            sv[p] = (uint16_t)rv[it];
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
            k[it] = sk[base + it * 32];
            rv[it] = sv[base + it * 32];
        }
    }
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        keys[base + it * 32] = k[it];
        vals[base + it * 32] = (int32_t)rv[it];
    }
    if (threadIdx.x == 0) plan[16] = 0;
}

// --------------------------------------------------------- K4 topology ----
__device__ __forceinline__ int lcp_levels(uint64_t a, uint64_t b, int D) {
    const uint64_t x = a ^ b;
    if (x == 0) return D;
    return (__clzll((long long)x) - (64 - 3 * D)) / 3;
}

struct TopoView {
    const uint64_t* keys;     // sorted
    const int32_t* vals;      // body index per sorted position
    const int32_t* depth;     // per body (input order)
    int n_in, n_total, D;
    int int_cap, cell_cap;    // capacities of the internal-node and cell arrays
    bool cut;                 // some path met a gap: depths differ from D
    // Bodies' depths are all D unless a path met a gap between float child
    // bounds (never in the batched form): only then are they gathered, two
    // random reads for every delta.
    __device__ void read_gaps(const int32_t* counters) { cut = counters[TC_GAPS] != 0; }
    __device__ int delta(int s) const {   // common levels of sorted bodies s and s+1; -1 past the end
        if (s < 0 || s + 1 >= n_in) return -1;
        int l = lcp_levels(keys[s], keys[s + 1], D);
        if (cut) {
            l = min(l, depth[vals[s]]);
            l = min(l, depth[vals[s + 1]]);
        }
        return l;
    }
    // Nodes starting at sorted position s: internal levels lo..hi and a leaf at
    // level lf (lf = -1: s lies inside an earlier bucket).
    __device__ void info(int s, int& lo, int& hi, int& nint, int& lf, int& cur) const {
        const int prev = (s > 0) ? delta(s - 1) : -1;
        cur = delta(s);
        if (prev >= D) { lo = 0; hi = -1; nint = 0; lf = -1; return; }
        lo = prev + 1;
        hi = min(cur, D - 1);
        if (s == 0 && n_total >= 2) hi = max(hi, 0);
        nint = max(0, hi - lo + 1);
        lf = nint > 0 ? hi + 1 : lo;
    }
};

__device__ __forceinline__ uint64_t node_code(uint64_t key, int level, int D) {
    return (1ull << (3 * level)) | (level ? (key >> (3 * (D - level))) : 0ull);
}

__device__ __forceinline__ uint32_t hash_slot(uint64_t code, uint32_t mask) {
    uint64_t x = code * 0x9E3779B97F4A7C15ull;
    x ^= x >> 29;
    return (uint32_t)x & mask;
}

__device__ void hash_insert(uint64_t* hk, int32_t* hv, uint32_t mask, uint64_t code, int32_t val, int32_t* counters) {
    uint32_t h = hash_slot(code, mask);
    for (uint32_t probe = 0; probe <= mask; ++probe) {
        const unsigned long long prev = atomicCAS((unsigned long long*)&hk[h], 0ull, (unsigned long long)code);
        if (prev == 0ull || prev == code) {
            hv[h] = val;
            return;
        }
        h = (h + 1) & mask;
    }
    atomicAdd(&counters[TC_HASHFAIL], 1);
}

__device__ int32_t hash_find(const uint64_t* hk, const int32_t* hv, uint32_t mask, uint64_t code, int32_t* counters) {
    uint32_t h = hash_slot(code, mask);
    for (uint32_t probe = 0; probe <= mask; ++probe) {
        const uint64_t k = hk[h];
        if (k == code) return hv[h];
        if (k == 0ull) break;
        h = (h + 1) & mask;
    }
    atomicAdd(&counters[TC_HASHFAIL], 1);
    return 0;
}

// Bounds of the node with the given code, replaying Octree::Split in float.
__device__ void node_bounds(uint64_t code, int level, float half, float3& lo, float3& hi, float& side) {
    lo = make_float3(-half, -half, -half);
    hi = make_float3(half, half, half);
    float size = __fsub_rn(hi.x, lo.x);
    for (int l = 1; l <= level; ++l) {
        const int dg = (int)((code >> (3 * (level - l))) & 7ull);
        const float s = __fmul_rn(size, 0.5f);   // Size / 2: exact halving, the same value as a division
        const float mx = __fadd_rn(lo.x, s), my = __fadd_rn(lo.y, s), mz = __fadd_rn(lo.z, s);
        if (dg & 1) { lo.x = mx; hi.x = __fadd_rn(mx, s); } else { hi.x = mx; }
        if (dg & 2) { lo.y = my; hi.y = __fadd_rn(my, s); } else { hi.y = my; }
        if (dg & 4) { lo.z = mz; hi.z = __fadd_rn(mz, s); } else { hi.z = mz; }
        size = __fsub_rn(hi.x, lo.x);
    }
    side = size;
}

// Positions in sorted order; brings the sort result to buffer 0 when the
// device plan left it in buffer 1 (no host read of the plan).  With curve, the
// last `curve` digits of the keys, sorted along the Hilbert curve, become octants
// again, those of a path that a gap cut (counters, depth; null where there are none)
// up to its end.
__global__ void __launch_bounds__(256) k_gather_final(const float4* pos, uint64_t* k0,
                                                      const uint64_t* k1, int32_t* v0,
                                                      const int32_t* v1, int n,
                                                      const int32_t* plan, float4* spos,
                                                      int curve, const int32_t* counters,
                                                      const int32_t* depth) {
    wait_for_previous();
    __shared__ uint32_t table[2 * kHilbertStates];
    if (curve) {   // uniform
        load_hilbert(table, true);
        __syncthreads();
    }
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const bool from1 = plan[16] != 0;
    const int v = from1 ? v1[s] : v0[s];
    if (curve) {
        const uint64_t key = from1 ? k1[s] : k0[s];
        const int d = counters && counters[TC_GAPS] != 0 && key != ~0ull ? depth[v] : curve;
        k0[s] = key == ~0ull ? key : hilbert_map_cut(key, d, curve, table);
    } else if (from1) {
        k0[s] = k1[s];
    }
    if (from1) v0[s] = v;
    spos[s] = (v >= 0 && v < n) ? pos[v] : make_float4(0.f, 0.f, 0.f, 0.f);
}

// Internal nodes and leaf starting at sorted position s; bucket size and
// whether a bucket's bodies differ.
__device__ __forceinline__ void position_nodes(const TopoView& tv, const float4* spos, int s, int& nint, int& lf,
                                               int& count, bool& deeper) {
    int lo, hi, cur;
    count = 0;
    deeper = false;
    if (s < tv.n_in) {
        tv.info(s, lo, hi, nint, lf, cur);
    } else {
        nint = 0; lf = -1; cur = -1;
    }
    if (lf >= 0) {
        count = 1;
        if (lf == tv.D && cur == tv.D) {
            int x = s;
            const float4 p0 = spos[s];
            while (x + 1 < tv.n_in && tv.delta(x) == tv.D) {
                ++x;
                ++count;
                const float4 q = spos[x];
                if (q.x != p0.x || q.y != p0.y || q.z != p0.z) deeper = true;
            }
        }
    }
}

// Per tile of kSortTile sorted positions: the nodes starting there, and the
// exclusive prefix of their internal-node counts by single-pass scan (pos_nint;
// the total goes to counters[TC_NINT]).  With hk_zero, the threads also clear
// the internal-node hash table for the emission that follows.  With
// host_counters (pinned), the last tile to finish sends the counters there.
//
// A thread takes every kPosThreads-th position (neighbouring threads read and
// write neighbouring words), and the counts go through shared memory to the
// scan, which wants consecutive ones.  Sixteen consecutive positions a thread and
// a depth gather for each delta took 81 us cold at 1M bodies; the whole topology
// phase went from 258 to 194 us there, from 98 to 73 us at 100,003 (events).
constexpr int kPosThreads = 1024;
constexpr int kPosItems = kSortTile / kPosThreads;
static_assert(kPosItems == 4, "the scan's counts are read as one int4 a thread");
__global__ void __launch_bounds__(kPosThreads) k_positions_scan(TopoView tv, const float4* spos,
                                                                int32_t* pos_nint,
                                                                int32_t* leaf_level,
                                                                int32_t* leaf_count,
                                                                int32_t* counters,
                                                                unsigned long long* status, int ntiles,
                                                                uint64_t* hk_zero, size_t hk_n,
                                                                int32_t* host_counters,
                                                                int* err) {
    wait_for_previous();
    __shared__ int sh_warp[33], sh_off, sh_tile, sh_leaf, sh_deeper;
    __shared__ __align__(16) int sh_nint[kSortTile];
    if (hk_zero)
        for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < hk_n; i += (size_t)gridDim.x * blockDim.x)
            hk_zero[i] = 0ull;
    if (threadIdx.x == 0) sh_leaf = sh_deeper = 0;
    const int tile = lb_tile_index(&counters[TC_TILE_POS], &sh_tile);
    tv.n_in = counters[TC_NIN];
    tv.read_gaps(counters);
    unsigned nleaf = 0, ndeeper = 0;
#pragma unroll
    for (int k = 0; k < kPosItems; ++k) {
        const int j = k * kPosThreads + threadIdx.x, s = tile * kSortTile + j;
        int nint = 0;
        if (s < tv.n_total) {
            int lf, count;
            bool deeper;
            position_nodes(tv, spos, s, nint, lf, count, deeper);
            leaf_level[s] = lf;
            leaf_count[s] = count;
            nleaf += lf >= 0 ? 1u : 0u;
            ndeeper += deeper ? 1u : 0u;
        }
        sh_nint[j] = nint;
    }
    nleaf = __reduce_add_sync(0xffffffffu, nleaf);
    ndeeper = __reduce_add_sync(0xffffffffu, ndeeper);
    if ((threadIdx.x & 31) == 0) {
        if (nleaf) atomicAdd(&sh_leaf, (int)nleaf);
        if (ndeeper) atomicAdd(&sh_deeper, (int)ndeeper);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (sh_leaf) atomicAdd(&counters[TC_NLEAF], sh_leaf);
        if (sh_deeper) atomicAdd(&counters[TC_DEEPER], sh_deeper);
    }
    int4* mine = reinterpret_cast<int4*>(sh_nint) + threadIdx.x;
    const int4 c = *mine;
    const int run = lb_scan_tile(c.x + c.y + c.z + c.w, tile, ntiles, status, counters + TC_NINT, sh_warp, &sh_off, err);
    *mine = make_int4(run, run + c.x, run + c.x + c.y, run + c.x + c.y + c.z);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPosItems; ++k) {
        const int j = k * kPosThreads + threadIdx.x, s = tile * kSortTile + j;
        if (s < tv.n_total) pos_nint[s] = sh_nint[j];
    }
    // (thread 0 made this tile's additions to the counters)
    if (host_counters && threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&counters[TC_DONE_POS], 1) == ntiles - 1) {
            __threadfence();
            for (int k = 0; k < TC_COUNT; ++k) host_counters[k] = __ldcg(counters + k);
        }
    }
}

// Emits the internal nodes starting at each sorted position (level, first
// body, code, hash entry) and clears their child mask and counters, and the
// look-back status of the child-count scan.
__global__ void k_emit(TopoView tv, const int32_t* int_base, int32_t* int_level,
                       int32_t* int_first, uint64_t* int_code, uint64_t* hk,
                       int32_t* hv, uint32_t hmask, uint32_t* int_mask,
                       int32_t* int_nint, int32_t* int_pending,
                       int32_t* counters, unsigned long long* popc_status,
                       int popc_tiles) {
    wait_for_previous();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    for (int i = s; i < popc_tiles; i += gridDim.x * blockDim.x) popc_status[i] = 0ull;   // for k_popc_scan
    tv.n_in = counters[TC_NIN];
    if (s >= tv.n_in) return;
    tv.read_gaps(counters);
    int lo, hi, nint, lf, cur;
    tv.info(s, lo, hi, nint, lf, cur);
    const uint64_t key = tv.keys[s];
    const int base = int_base[s];
    for (int l = lo; l <= hi; ++l) {
        const int k = base + (l - lo);
        if (k >= tv.int_cap) {
            atomicAdd(&counters[TC_OVERFLOW], 1);
            break;
        }
        const uint64_t code = node_code(key, l, tv.D);
        int_level[k] = l;
        int_first[k] = s;
        int_code[k] = code;
        int_mask[k] = 0u;
        int_nint[k] = 0;
        int_pending[k] = 0;
        hash_insert(hk, hv, hmask, code, k, counters);
    }
}

__device__ __forceinline__ void link_internal(int k, const int32_t* int_level,
                                              const int32_t* int_first,
                                              const uint64_t* int_code, const TopoView& tv, int ni,
                                              const uint64_t* hk, const int32_t* hv,
                                              uint32_t hmask, int32_t* int_parent,
                                              uint32_t* int_mask, int32_t* int_nint,
                                              int32_t* counters) {
    if (k >= ni || k == 0) return;
    const int l = int_level[k];
    const int s = int_first[k];
    const uint64_t code = int_code[k];
    const int prev = (s > 0) ? tv.delta(s - 1) : -1;
    const int parent = (l > prev + 1) ? k - 1 : hash_find(hk, hv, hmask, code >> 3, counters);
    if (parent < 0 || parent >= ni) {
        atomicAdd(&counters[TC_OVERFLOW], 1);
        return;
    }
    int_parent[k] = parent;
    atomicOr(&int_mask[parent], 1u << (unsigned)(code & 7ull));
    atomicAdd(&int_nint[parent], 1);
}

__device__ __forceinline__ void link_leaf(int s, const TopoView& tv, const int32_t* int_base,
                                          const int32_t* leaf_level, const uint64_t* hk,
                                          const int32_t* hv, uint32_t hmask,
                                          int32_t* leaf_parent, uint32_t* int_mask,
                                          int32_t* counters) {
    if (s >= tv.n_in) return;
    const int lf = leaf_level[s];
    if (lf <= 0) return;
    int lo, hi, nint, lf2, cur;
    tv.info(s, lo, hi, nint, lf2, cur);
    const uint64_t code = node_code(tv.keys[s], lf, tv.D);
    const int parent = nint > 0 ? int_base[s] + (lf - 1 - lo) : hash_find(hk, hv, hmask, code >> 3, counters);
    if (parent < 0 || parent >= tv.int_cap) {
        atomicAdd(&counters[TC_OVERFLOW], 1);
        return;
    }
    leaf_parent[s] = parent;
    atomicOr(&int_mask[parent], 1u << (unsigned)(code & 7ull));
}

// Every node's parent and the parents' child masks: blocks [0, int_blocks)
// link internal nodes, the rest link the leaf starting at each position.
// n_int_dev (graph builds) bounds the internal nodes by the device count.
__global__ void k_link(const int32_t* int_level, const int32_t* int_first,
                       const uint64_t* int_code, TopoView tv, int n_int,
                       const int32_t* n_int_dev, int int_blocks, const int32_t* int_base,
                       const int32_t* leaf_level, const uint64_t* hk,
                       const int32_t* hv, uint32_t hmask, int32_t* int_parent,
                       int32_t* leaf_parent, uint32_t* int_mask,
                       int32_t* int_nint, int32_t* counters) {
    wait_for_previous();
    tv.read_gaps(counters);
    if ((int)blockIdx.x < int_blocks) {
        const int k = blockIdx.x * blockDim.x + threadIdx.x;
        const int ni = n_int_dev ? min(*n_int_dev, n_int) : n_int;
        link_internal(k, int_level, int_first, int_code, tv, ni, hk, hv, hmask, int_parent, int_mask, int_nint,
                      counters);
    } else {
        const int s = (blockIdx.x - int_blocks) * blockDim.x + threadIdx.x;
        link_leaf(s, tv, int_base, leaf_level, hk, hv, hmask, leaf_parent, int_mask, counters);
    }
}

// int_block[k] = non-empty children of internal nodes before k (their first
// child cell, less one), by single-pass scan over tiles of kSortTile nodes
// (the layout of k_positions_scan).
__global__ void __launch_bounds__(kPosThreads) k_popc_scan(const uint32_t* mask, int n_int,
                                                            const int32_t* n_int_dev,
                                                            int32_t* out, int32_t* counters,
                                                            unsigned long long* status, int ntiles,
                                                            int* err) {
    wait_for_previous();
    __shared__ int sh_warp[33], sh_off, sh_tile;
    const int tile = lb_tile_index(&counters[TC_TILE_POPC], &sh_tile);
    const int ni = n_int_dev ? min(*n_int_dev, n_int) : n_int;
    __shared__ __align__(16) int sh_cnt[kSortTile];
#pragma unroll
    for (int k = 0; k < kPosItems; ++k) {
        const int j = k * kPosThreads + threadIdx.x, q = tile * kSortTile + j;
        sh_cnt[j] = q < ni ? __popc(mask[q]) : 0;
    }
    __syncthreads();
    int4* mine = reinterpret_cast<int4*>(sh_cnt) + threadIdx.x;
    const int4 c = *mine;
    const int run = lb_scan_tile(c.x + c.y + c.z + c.w, tile, ntiles, status, nullptr, sh_warp, &sh_off, err);
    *mine = make_int4(run, run + c.x, run + c.x + c.y, run + c.x + c.y + c.z);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPosItems; ++k) {
        const int j = k * kPosThreads + threadIdx.x, q = tile * kSortTile + j;
        if (q < n_int) out[q] = sh_cnt[j];
    }
}

// Opening thresholds of a cell for the traversal: with r^2 computed exactly
// as the reference does, r^2 > accept_r2 guarantees float(side / r) < theta_f
// and r^2 < reject_r2 guarantees the opposite (1e-5 relative margins, far
// above the float rounding of the ratio); between the two the traversal
// evaluates the exactly rounded ratio.
__device__ __forceinline__ void open_thresholds(float side, float theta_f, int& accept_bits, int& reject_bits) {
    const double q = (double)side * (double)side / ((double)theta_f * (double)theta_f);
    accept_bits = __float_as_int(__double2float_ru(q * (1.0 + 1e-5)));
    reject_bits = __float_as_int(__double2float_rd(q * (1.0 - 1e-5)));
}

__device__ __forceinline__ int child_cell(const int32_t* int_block, const uint32_t* int_mask, int parent, int oct) {
    return 1 + int_block[parent] + __popc(int_mask[parent] & ((1u << oct) - 1u));
}

__device__ __forceinline__ void place_internal(int k, const int32_t* int_level,
                                               const uint64_t* int_code,
                                               const int32_t* int_parent,
                                               const uint32_t* int_mask,
                                               const int32_t* int_block, int ni, int cell_cap,
                                               float half, float theta_f, int32_t* int_cell,
                                               int4* cell_meta, float4* cell_lo,
                                               float4* cell_hi, uint64_t* cell_code,
                                               bool batch) {
    if (k >= ni) return;
    const uint64_t code = int_code[k];
    const int l = int_level[k];
    const int cell = (k == 0) ? 0 : child_cell(int_block, int_mask, int_parent[k], (int)(code & 7ull));
    if (cell >= cell_cap) {
        int_cell[k] = 0;
        return;
    }
    int_cell[k] = cell;
    if (batch) return;   // the batched form's moment pass writes the node's record
    float3 lo, hi;
    float side;
    node_bounds(code, l, half, lo, hi, side);
    const uint32_t m = int_mask[k];
    int ab, rb;
    open_thresholds(side, theta_f, ab, rb);
    cell_meta[cell] = make_int4(1 + int_block[k], ab, rb, KIND_INTERNAL | (__popc(m) << 4));
    cell_lo[cell] = make_float4(lo.x, lo.y, lo.z, side);
    cell_hi[cell] = make_float4(hi.x, hi.y, hi.z, (float)l);
    cell_code[cell] = code;
}

__device__ __forceinline__ void place_leaf(int s, const TopoView& tv, const int32_t* leaf_level,
                                           const int32_t* leaf_count,
                                           const int32_t* leaf_parent,
                                           const uint32_t* int_mask,
                                           const int32_t* int_block, const float4* spos,
                                           float half, float theta_f, float4* cell_com,
                                           double* cell_mass, int32_t* cell_count,
                                           int4* cell_meta, float4* cell_lo,
                                           float4* cell_hi, uint64_t* cell_code,
                                           CellRec* rec) {
    if (s >= tv.n_in) return;
    const int lf = leaf_level[s];
    if (lf < 0) return;
    const uint64_t code = node_code(tv.keys[s], lf, tv.D);
    if (lf > 0 && (leaf_parent[s] < 0 || leaf_parent[s] >= tv.int_cap)) return;   // parent lost to an overflow
    const int cell = (lf == 0) ? 0 : child_cell(int_block, int_mask, leaf_parent[s], (int)(code & 7ull));
    if (cell >= tv.cell_cap) return;
    if (rec) {   // the batched form: the leaf's whole record (bodies clamped to the sorted range)
        write_leaf_record(rec + cell, spos, s, max(1, min(leaf_count[s], tv.n_in - s)), lf);
        return;
    }
    float3 lo, hi;
    float side;
    node_bounds(code, lf, half, lo, hi, side);
    const int count = leaf_count[s];
    float4 com;
    double M;
    if (count == 1) {
        // leaf with one body: CentreOfMass = P->Position, TotalMass = P->Mass
        com = spos[s];
        M = (double)com.w;
    } else {
        // depth-cap bucket: bodies in ascending index order
        float cx = 0.f, cy = 0.f, cz = 0.f;
        M = 0.0;
        for (int q = s; q < s + count; ++q) {
            const float4 p = spos[q];
            M += (double)p.w;
            const float mf = p.w;
            cx = __fadd_rn(cx, __fmul_rn(p.x, mf));
            cy = __fadd_rn(cy, __fmul_rn(p.y, mf));
            cz = __fadd_rn(cz, __fmul_rn(p.z, mf));
        }
        if (M > 0.0) {
            const float inv = __fdiv_rn(1.0f, (float)M);
            cx = __fmul_rn(cx, inv); cy = __fmul_rn(cy, inv); cz = __fmul_rn(cz, inv);
        }
        com = make_float4(cx, cy, cz, (float)M);
    }
    com.w = (float)M;
    cell_com[cell] = com;
    cell_mass[cell] = M;
    int ab, rb;
    open_thresholds(side, theta_f, ab, rb);
    cell_meta[cell] = make_int4(s, ab, rb, (count == 1 ? KIND_SINGLE : KIND_BUCKET) | (count << 8));
    cell_count[cell] = count;
    cell_lo[cell] = make_float4(lo.x, lo.y, lo.z, side);
    cell_hi[cell] = make_float4(hi.x, hi.y, hi.z, (float)lf);
    cell_code[cell] = code;
}

// Every cell: blocks [0, int_blocks) place internal nodes (bounds, opening
// thresholds, first child), the rest the leaf starting at each position
// (bounds, thresholds, mass and centre of mass of its body or bucket).  With
// rec (the batched form) an internal node only gets its cell and a leaf its
// 64-byte record.
__global__ void k_place(const int32_t* int_level, const uint64_t* int_code,
                        const int32_t* int_parent, const uint32_t* int_mask,
                        const int32_t* int_block, int n_int, const int32_t* n_int_dev,
                        int int_blocks, TopoView tv, const int32_t* leaf_level,
                        const int32_t* leaf_count, const int32_t* leaf_parent,
                        const float4* spos, float half, float theta_f, int32_t* int_cell,
                        float4* cell_com, double* cell_mass,
                        int32_t* cell_count, int4* cell_meta, float4* cell_lo,
                        float4* cell_hi, uint64_t* cell_code, CellRec* rec) {
    wait_for_previous();
    if ((int)blockIdx.x < int_blocks) {
        const int k = blockIdx.x * blockDim.x + threadIdx.x;
        const int ni = n_int_dev ? min(*n_int_dev, n_int) : n_int;
        place_internal(k, int_level, int_code, int_parent, int_mask, int_block, ni, tv.cell_cap, half, theta_f,
                       int_cell, cell_meta, cell_lo, cell_hi, cell_code, rec != nullptr);
    } else {
        const int s = (blockIdx.x - int_blocks) * blockDim.x + threadIdx.x;
        place_leaf(s, tv, leaf_level, leaf_count, leaf_parent, int_mask, int_block, spos, half, theta_f, cell_com,
                   cell_mass, cell_count, cell_meta, cell_lo, cell_hi, cell_code, rec);
    }
}

// ------------------------------------------------------------- K5 mass ----
// One thread starts at each internal node whose children are all leaves; the
// last child of a node to arrive finishes it.  The bound is the chain of
// memory round trips from the deepest node to the root, so a level costs as few
// as it can: all the children are read at once (eight predicated loads, not a
// loop of dependent ones), a node's own words are read while its arrival
// counter is on the way, and a node with a single child (the levels between
// the root cube and a small galaxy, and those above close pairs) is finished
// from registers.  Events: 34 -> 24 us at 4,000 bodies, 57 -> 37 at 100,003,
// 123 -> 105 at 1M, where the scattered cells of a million bodies bound it.
struct NodeMass {
    double M;
    float cx, cy, cz;
    int count;
};

__device__ __forceinline__ void scale_com(NodeMass& m) {
    if (m.M > 0.0) {
        const float inv = __fdiv_rn(1.0f, (float)m.M);
        m.cx = __fmul_rn(m.cx, inv); m.cy = __fmul_rn(m.cy, inv); m.cz = __fmul_rn(m.cz, inv);
    }
}

// Children of the node whose first child cell is F.
__device__ __forceinline__ NodeMass sum_children(int F, int nch, const float4* cell_com, const double* cell_mass,
                                                 const int32_t* cell_count) {
    double mc[8];
    float4 cc[8];
    int cnt[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (j < nch) {
            mc[j] = load_published(&cell_mass[F + j]);
            cc[j] = load_published(&cell_com[F + j]);
            cnt[j] = load_published(&cell_count[F + j]);
        }
    }
    NodeMass m{0.0, 0.f, 0.f, 0.f, 0};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (j < nch) {
            m.M += mc[j];
            const float mf = (float)mc[j];
            m.cx = __fadd_rn(m.cx, __fmul_rn(cc[j].x, mf));
            m.cy = __fadd_rn(m.cy, __fmul_rn(cc[j].y, mf));
            m.cz = __fadd_rn(m.cz, __fmul_rn(cc[j].z, mf));
            m.count += cnt[j];
        }
    }
    scale_com(m);
    return m;
}

__global__ void __launch_bounds__(128) k_mass(int n_int, const int32_t* int_parent,
                                              const int32_t* int_nint, int32_t* int_pending,
                                              const int32_t* int_cell,
                                              const int32_t* int_block,
                                              const uint32_t* int_mask, float4* cell_com,
                                              double* cell_mass, int32_t* cell_count,
                                              int dropped) {
    wait_for_previous();
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_int || int_nint[k] != 0) return;
    int cell = int_cell[k], parent = k > 0 ? int_parent[k] : 0;
    NodeMass m = sum_children(1 + int_block[k], __popc(int_mask[k]), cell_com, cell_mass, cell_count);
    for (int guard = 0; guard < 64; ++guard) {   // a path has at most 22 internal nodes
        if (k == 0) m.count += dropped;
        __stcg(&cell_com[cell], make_float4(m.cx, m.cy, m.cz, (float)m.M));
        __stcg(&cell_mass[cell], m.M);
        __stcg(&cell_count[cell], m.count);
        if (k == 0) return;
        const int p = parent;
        const int nint = int_nint[p], first = 1 + int_block[p], nch = __popc(int_mask[p]);
        cell = int_cell[p];
        parent = p > 0 ? int_parent[p] : 0;
        if (nch == 1) {   // the only child: its sums are in registers
            const float mf = (float)m.M;
            // 0 + x as the sum over children starts: a negative zero becomes +0 there too
            m.M = 0.0 + m.M;
            m.cx = __fadd_rn(0.f, __fmul_rn(m.cx, mf));
            m.cy = __fadd_rn(0.f, __fmul_rn(m.cy, mf));
            m.cz = __fadd_rn(0.f, __fmul_rn(m.cz, mf));
            scale_com(m);
        } else {
            if (nint > 1) {
                const int old = atomic_add_acq_rel(&int_pending[p], 1);   // publishes this node, sees its siblings
                if (old != nint - 1) return;
            }
            // (with one internal child the siblings are leaves, complete since the placement)
            m = sum_children(first, nch, cell_com, cell_mass, cell_count);
        }
        k = p;
    }
}

// ------------------------------------------------- batched forest keys ----
// Keys of the batched form's Barnes-Hut bodies [0, n) (nb_morton.cuh, the
// position's digits in Hilbert order), with
// the radix sort's histograms and the look-back status cleared,
// kSortThreads * items keys a block; the first threads also write each galaxy's cube for the
// traversal.  Pad entries [n, tiles * kSortTile) get key ~0.
__global__ void __launch_bounds__(kSortThreads) k_batch_keys_hist(
    const float4* __restrict__ pos, const int32_t* __restrict__ body_slot, int n, const unsigned* __restrict__ box_bits,
    int nslot, float4* __restrict__ gal_box, uint64_t* __restrict__ keys, int32_t* __restrict__ vals,
    int32_t* __restrict__ depth, uint32_t* __restrict__ ghist, unsigned long long* __restrict__ sort_status,
    int ntiles, unsigned long long* __restrict__ pos_status, int items, int key_blocks) {
    __shared__ uint32_t table[2 * kHilbertStates];
    __shared__ uint32_t h[kPasses][256];
    __shared__ unsigned long long sh_groups[2 * kKeyGroups];
    const int g = blockIdx.x * kSortThreads + threadIdx.x;
    if (g < nslot) gal_box[g] = gal_cube(box_bits, g);
    if ((int)blockIdx.x >= key_blocks) return;   // blocks past the keys only write galaxy cubes (block-uniform)
    for (int i = threadIdx.x; i < kPasses * 256; i += kSortThreads) (&h[0][0])[i] = 0;
    if (threadIdx.x < 2 * kKeyGroups) sh_groups[threadIdx.x] = 0ull;
    load_hilbert(table, false);
    zero_tile_status(sort_status, ntiles, pos_status, key_blocks);
    __syncthreads();
    for (int it = 0; it < items; ++it) {
        const int i = (blockIdx.x * items + it) * kSortThreads + threadIdx.x;
        vals[i] = i;
        uint64_t key = ~0ull;
        if (i < n) {
            const int slot = body_slot[i];
            key = hilbert_map(forest_key(pos[i], slot, gal_cube(box_bits, slot)), kMortonLevels, table);
            depth[i] = kBatchDepth;
        }
        keys[i] = key;
        count_key(key, h, sh_groups);
    }
    flush_hist(h, sh_groups, ghist);
}

// --------------------------------------------------------------- host ----
// Replaces *p by a buffer of `bytes` (the old one returned after the work
// queued on st).
static cudaError_t grow(void** p, size_t bytes, cudaStream_t st) {
    dev_free(*p, st);
    *p = nullptr;
    return dev_alloc(p, bytes);
}

#define NB_TRY(x)                               \
    do {                                        \
        cudaError_t e_ = (x);                   \
        if (e_ != cudaSuccess) return e_;       \
    } while (0)

static cudaError_t reserve_bodies(nb_sim* sim, size_t nk) {
    TreeBuffers& t = sim->tree;
    if (nk <= t.body_cap) return cudaSuccess;
    const size_t cap = nk;
    t.body_cap = 0;   // until every array is there
    NB_TRY(grow((void**)&t.keys[0], cap * 8, sim->stream));
    NB_TRY(grow((void**)&t.keys[1], cap * 8, sim->stream));
    NB_TRY(grow((void**)&t.vals[0], cap * 4, sim->stream));
    NB_TRY(grow((void**)&t.vals[1], cap * 4, sim->stream));
    NB_TRY(grow((void**)&t.depth, cap * 4, sim->stream));
    NB_TRY(grow((void**)&t.spos, cap * 16, sim->stream));
    NB_TRY(grow((void**)&t.pos_nint, cap * 4, sim->stream));
    NB_TRY(grow((void**)&t.leaf_level, cap * 4, sim->stream));
    NB_TRY(grow((void**)&t.leaf_count, cap * 4, sim->stream));
    NB_TRY(grow((void**)&t.leaf_parent, cap * 4, sim->stream));
    const size_t ntiles = cap / kSortTile;
    NB_TRY(grow((void**)&t.sort_status, (size_t)kPasses * ntiles * 256 * sizeof(unsigned long long), sim->stream));
    NB_TRY(grow((void**)&t.pos_status, ntiles * sizeof(unsigned long long), sim->stream));
    if (!t.plan) NB_TRY(dev_alloc(&t.plan, 32 * 4));
    if (!t.dig_off) NB_TRY(dev_alloc(&t.dig_off, kPasses * 256 * 4));
    if (!t.counters) {
        // counters, tile counters of the look-back kernels, then the radix histograms
        NB_TRY(dev_alloc(&t.counters, (kCounterWords + kPasses * 256 + 4 * kKeyGroups) * 4));
        t.ghist = reinterpret_cast<uint32_t*>(t.counters + kCounterWords);
    }
    if (!t.h_counters) NB_TRY(cudaMallocHost(&t.h_counters, TC_COUNT * 4));
    if (!t.counted) NB_TRY(cudaEventCreateWithFlags(&t.counted, cudaEventDisableTiming));
    if (!t.interactions) NB_TRY(dev_alloc(&t.interactions, sizeof(unsigned long long)));
    t.body_cap = cap;
    return cudaSuccess;
}

static cudaError_t reserve_nodes(nb_sim* sim, size_t n_int, size_t n_cells) {
    return grow_nodes(sim->tree, n_int, n_cells, (size_t)kSortTile,
                      [sim](void** p, size_t bytes) { return grow(p, bytes, sim->stream); });
}

cudaError_t tree_reserve(nb_sim* sim) {
    return reserve_bodies(sim, pad_up(std::max<size_t>(sim->n, 1), kSortTile));
}

void tree_free(nb_sim* sim) {
    TreeBuffers& t = sim->tree;
    void* ptrs[] = {t.keys[0], t.keys[1], t.vals[0], t.vals[1], t.depth, t.spos, t.pos_nint, t.leaf_level,
                    t.leaf_count, t.leaf_parent, t.int_level, t.int_first, t.int_parent, t.int_mask, t.int_nint,
                    t.int_pending, t.int_block, t.int_cell, t.int_code, t.cell_com, t.cell_meta, t.cell_mass,
                    t.cell_lo, t.cell_hi, t.cell_code, t.cell_count, t.hkeys, t.hvals, t.sort_status, t.pos_status,
                    t.popc_status, t.dig_off, t.plan, t.counters, t.interactions};
    for (void* p : ptrs) dev_free(p, sim->stream);
    if (t.h_counters) cudaFreeHost(t.h_counters);
    if (t.counted) cudaEventDestroy(t.counted);
    t = TreeBuffers{};
}

float theta_float(double theta) {
    float f = (float)theta;
    if ((double)f < theta) f = std::nextafter(f, INFINITY);
    return f;
}

static TopoView topo_view(nb_sim* sim) {
    TreeBuffers& t = sim->tree;
    TopoView tv;
    tv.keys = t.keys[t.final_buf];
    tv.vals = t.vals[t.final_buf];
    tv.depth = t.depth;
    tv.n_in = t.n_in;
    tv.n_total = (int)sim->n;
    tv.D = sim->prm.max_depth;
    tv.int_cap = (int)t.int_cap;
    tv.cell_cap = (int)t.cell_cap;
    tv.cut = true;   // read_gaps in the kernels
    return tv;
}

// Clears the counters and histograms, then keys of the current positions into
// t.keys[0] (input order, t.vals[0] = identity) with their histograms.
static cudaError_t launch_keys(nb_sim* sim, size_t nk, bool curve) {
    TreeBuffers& t = sim->tree;
    const int ntiles = (int)(nk / kSortTile);
    NB_TRY(cudaMemsetAsync(t.counters, 0, (kCounterWords + kPasses * 256 + 4 * kKeyGroups) * 4, sim->stream));
    PhaseScope ps(sim, NB_PHASE_KEYS);
    const int items = keys_per_thread(nk, sim->sm_count);
    k_keys_hist<<<(unsigned)(nk / (size_t)(kSortThreads * items)), kSortThreads, 0, sim->stream>>>(
        sim->pos, (int)sim->n, sim->prm.bounds_half, sim->prm.max_depth, t.keys[0], t.vals[0], t.depth, t.counters,
        t.ghist, t.sort_status, ntiles, t.pos_status, items, curve);
    return cudaGetLastError();
}

static cudaError_t launch_sort_block(TreeBuffers& t, cudaStream_t st) {
    // (set on each call: cheap, and right for every device)
    const cudaError_t e = cudaFuncSetAttribute(k_sort_block, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)kOneBytes);
    if (e != cudaSuccess) return e;
    NB_TRY(launch_after(k_sort_block, 1, kOneThreads, kOneBytes, st, t.keys[0], t.vals[0],
                        t.ghist, t.plan));
    return cudaGetLastError();
}

// The radix sort of t.keys[0] / t.vals[0] (histograms already made): one tile
// in one block, else the device plan, then one launch per pass.
static cudaError_t launch_sort(nb_sim* sim, size_t nk) {
    TreeBuffers& t = sim->tree;
    const int ntiles = (int)(nk / kSortTile);
    cudaStream_t st = sim->stream;
    if (ntiles == 1) {
        PhaseScope ps(sim, NB_PHASE_SORT);
        return launch_sort_block(t, st);
    }
    PhaseScope ps(sim, NB_PHASE_SORT, 1 + kPasses);
    NB_TRY(launch_after(k_sort_plan, 1, 256, 0, st, t.ghist, (int)nk, t.plan, t.dig_off));
    for (int p = 0; p < kPasses; ++p)
        NB_TRY(launch_after(k_sort_pass, ntiles, kPassThreads, 0, st, t.keys[0], t.keys[1], t.vals[0], t.vals[1],
                            ntiles, t.plan, p, t.dig_off, t.sort_status + (size_t)p * ntiles * 256,
                            t.counters + TC_TILE_SORT + p, sim->d_err));
    return cudaGetLastError();
}

// The emission into the node arrays as they are (bodies inside the root: counted
// on the device).
static cudaError_t launch_emit(nb_sim* sim, const TopoView& tv) {
    TreeBuffers& t = sim->tree;
    return launch_after(k_emit, (unsigned)((sim->n + kEmitBlock - 1) / kEmitBlock), kEmitBlock, 0, sim->stream, tv,
                        t.pos_nint, t.int_level, t.int_first, t.int_code, t.hkeys, t.hvals, (uint32_t)(t.hash_cap - 1),
                        t.int_mask, t.int_nint, t.int_pending, t.counters, t.popc_status,
                        (int)((t.int_cap + kSortTile - 1) / kSortTile));
}

cudaError_t tree_build(nb_sim* sim, bool export_order) {
    TreeBuffers& t = sim->tree;
    const int n = (int)sim->n;
    // Bodies along the Hilbert curve for a force pass: its groups of 64 consecutive
    // bodies are compact (in Morton order a run often jumps between cells that do not
    // touch), so fewer cells are decided body by body or taken by part of a group.
    // The traversal at 1,048,576 bodies took 3.04 ms instead of 3.58, at 100,003
    // 0.43 instead of 0.62; the keys' map costs 9 us and 1 us.
    const bool curve = !export_order;
    const size_t nk = pad_up(std::max<size_t>(sim->n, 1), kSortTile);
    const int ntiles = (int)(nk / kSortTile);
    NB_TRY(tree_reserve(sim));
    cudaStream_t st = sim->stream;
    // Every launch up to the traversal is a programmatic dependent launch
    // (nb_common.cuh): up to 17 dependent kernels, most of 3 to 40 us, whose gaps
    // added up.  A step of 4000 bodies 155 -> 143 us, of 100,003 639 -> 600, of 2^20
    // 3552 -> 3514.
    NB_TRY(launch_keys(sim, nk, curve));
    NB_TRY(launch_sort(sim, nk));
    bool early = false;
    // The sort result's buffer is decided on the device (passes with a constant
    // digit are skipped): the gather brings it to buffer 0 when it ended in
    // buffer 1, so no host read is needed here.
    {
        PhaseScope ps(sim, NB_PHASE_TOPOLOGY, t.int_cap > 0 ? 3 : 2);
        NB_TRY(launch_after(k_gather_final, (n + 255) / 256, 256, 0, st, sim->pos, t.keys[0], t.keys[1], t.vals[0],
                            t.vals[1], n, t.plan, t.spos, curve ? sim->prm.max_depth : 0, t.counters, t.depth));
        t.final_buf = 0;
        TopoView tv = topo_view(sim);
        // The scan clears the hash table as it stands and sends the counters to the
        // host itself: a copy before the wait and a memset behind it
        // took 5 us more of the phase at 4000 bodies (52 now), 8 at 2^20 (192).
        NB_TRY(launch_after(k_positions_scan, ntiles, kPosThreads, 0, st, tv, t.spos, t.pos_nint, t.leaf_level,
                            t.leaf_count, t.counters, t.pos_status, ntiles, t.int_cap > 0 ? t.hkeys : nullptr, t.hash_cap,
                            t.h_counters, sim->d_err));
        NB_TRY(cudaEventRecord(t.counted, st));
        // While the host waits for the counts, the nodes are emitted into the arrays
        // as they are; if they turn out too small, again into larger ones.
        // (The GPU idled here: the topology phase of 4000 bodies took 47 us, now 42, of
        // 100,003 57 and 51; a 4000-body frame 145 and 137.)
        early = t.int_cap > 0;
        if (early) NB_TRY(launch_emit(sim, tv));
        NB_TRY(cudaEventSynchronize(t.counted));
    }
    t.n_in = t.h_counters[TC_NIN];
    t.n_int = t.h_counters[TC_NINT];
    t.n_cells = t.n_int + t.h_counters[TC_NLEAF];
    t.trivial = (n < 2) || (t.n_in < 2 && t.n_int == 0) || t.n_in == 0;
    t.curve = curve;
    if (t.trivial) return cudaSuccess;
    const size_t cleared = t.int_cap;
    NB_TRY(reserve_nodes(sim, (size_t)t.n_int, (size_t)t.n_cells));
    const bool grown = t.int_cap != cleared;
    if (grown) {   // the arrays come with a new table, of the same size or not
        NB_TRY(cudaMemsetAsync(t.hkeys, 0, t.hash_cap * 8, st));
        if (early) NB_TRY(cudaMemsetAsync(t.counters + TC_OVERFLOW, 0, sizeof(int32_t), st));
    }
    TopoView tv = topo_view(sim);
    const int ni = t.n_int;
    const float tf = theta_float(sim->prm.theta);
    const uint32_t hmask = (uint32_t)(t.hash_cap - 1);
    {
        PhaseScope ps(sim, NB_PHASE_TOPOLOGY, grown || !early ? 4 : 3);
        const int nbk = (t.n_in + kEmitBlock - 1) / kEmitBlock;
        const int ib = (ni + kEmitBlock - 1) / kEmitBlock;
        const int ptiles = (ni + kSortTile - 1) / kSortTile;
        if (grown || !early) NB_TRY(launch_emit(sim, tv));
        NB_TRY(launch_after(k_link, ib + nbk, kEmitBlock, 0, st, t.int_level, t.int_first, t.int_code, tv, ni,
                            nullptr, ib, t.pos_nint, t.leaf_level, t.hkeys, t.hvals, hmask, t.int_parent,
                            t.leaf_parent, t.int_mask, t.int_nint, t.counters));
        NB_TRY(launch_after(k_popc_scan, ptiles, kPosThreads, 0, st, t.int_mask, ni, nullptr, t.int_block,
                            t.counters, t.popc_status, ptiles, sim->d_err));
        NB_TRY(launch_after(k_place, ib + nbk, kEmitBlock, 0, st, t.int_level, t.int_code, t.int_parent, t.int_mask,
                            t.int_block, ni, nullptr, ib, tv, t.leaf_level, t.leaf_count, t.leaf_parent, t.spos,
                            sim->prm.bounds_half, tf, t.int_cell, t.cell_com, t.cell_mass, t.cell_count,
                            t.cell_meta, t.cell_lo, t.cell_hi, t.cell_code, nullptr));
        NB_TRY(cudaGetLastError());
    }
    {
        PhaseScope ps(sim, NB_PHASE_MASS);
        NB_TRY(launch_after(k_mass, (ni + 127) / 128, 128, 0, st, ni, t.int_parent, t.int_nint, t.int_pending,
                            t.int_cell, t.int_block, t.int_mask, t.cell_com, t.cell_mass, t.cell_count,
                            n - t.n_in));
        NB_TRY(cudaGetLastError());
    }
    sim->tree_valid = true;
    return cudaSuccess;
}

cudaError_t tree_sizes(nb_sim* sim, int32_t* cells, int32_t* internal) {
    if (cells) *cells = sim->tree.trivial ? 0 : sim->tree.n_cells;
    if (internal) *internal = sim->tree.trivial ? 0 : sim->tree.n_int;
    return cudaSuccess;
}

// Keys of the current positions in input order (for export).
cudaError_t tree_keys_export(nb_sim* sim, uint64_t* d_keys, int32_t* d_depth) {
    TreeBuffers& t = sim->tree;
    const size_t nk = pad_up(std::max<size_t>(sim->n, 1), kSortTile);
    NB_TRY(tree_reserve(sim));
    NB_TRY(launch_keys(sim, nk, false));
    NB_TRY(cudaMemcpyAsync(d_keys, t.keys[0], sim->n * 8, cudaMemcpyDeviceToDevice, sim->stream));
    NB_TRY(cudaMemcpyAsync(d_depth, t.depth, sim->n * 4, cudaMemcpyDeviceToDevice, sim->stream));
    sim->tree_valid = false;   // the sort buffers no longer match the tree
    return cudaSuccess;
}

}  // namespace nb

// ----------------------------------------------------------------------------
// Topology without host synchronisation, for the batched form (its steps are
// captured in a CUDA graph).  The batched step's first kernel clears the
// counters and histograms and sets TC_NIN = n; tree_batch_keys writes the
// keys of bodies [0, n), their histograms and clears the look-back status
// (every body lies inside its cube).  Grid sizes come from the capacities;
// the kernels read the node counts on the device and report overflow in
// counters[TC_OVERFLOW].
// ----------------------------------------------------------------------------
namespace nb {

int tree_counter_words() { return kCounterWords + kPasses * 256 + 4 * kKeyGroups; }

cudaError_t tree_batch_keys(nb_sim* sim, const float4* pos, const int32_t* body_slot, int n,
                            const unsigned* box_bits, int nslot, float4* gal_box) {
    TreeBuffers& t = sim->tree;
    const size_t nk = pad_up(std::max<size_t>((size_t)n, 1), kSortTile);
    const int ntiles = (int)(nk / kSortTile);
    const int items = keys_per_thread(nk, sim->sm_count);
    const int key_blocks = (int)(nk / (size_t)(kSortThreads * items));
    const int blocks = std::max(key_blocks, (nslot + kSortThreads - 1) / kSortThreads);
    PhaseScope ps(sim, NB_PHASE_KEYS);
    k_batch_keys_hist<<<blocks, kSortThreads, 0, sim->stream>>>(pos, body_slot, n, box_bits, nslot, gal_box,
                                                                t.keys[0], t.vals[0], t.depth, t.ghist,
                                                                t.sort_status, ntiles, t.pos_status, items,
                                                                key_blocks);
    return cudaGetLastError();
}

cudaError_t tree_build_graph(nb_sim* sim, const float4* pos, int n, int D, bool counts_only, CellRec* rec) {
    TreeBuffers& t = sim->tree;
    const size_t nk = pad_up(std::max<size_t>((size_t)n, 1), kSortTile);
    const int ntiles = (int)(nk / kSortTile);
    cudaStream_t st = sim->stream;
    if (!counts_only && t.int_cap == 0) return cudaErrorMemoryAllocation;   // the node arrays were not to be had
    NB_TRY(launch_sort(sim, nk));
    t.final_buf = 0;
    t.n_in = n;
    TopoView tv;
    tv.keys = t.keys[0];
    tv.vals = t.vals[0];
    tv.depth = t.depth;
    tv.n_in = n;
    tv.n_total = n;
    tv.D = D;
    tv.int_cap = (int)t.int_cap;
    tv.cell_cap = (int)t.cell_cap;
    tv.cut = true;   // read_gaps in the kernels
    const int icap = (int)t.int_cap;
    const uint32_t hmask = (uint32_t)(t.hash_cap - 1);
    const int nbk = (n + kEmitBlock - 1) / kEmitBlock;
    const int ib = (icap + kEmitBlock - 1) / kEmitBlock;
    const int ptiles = (icap + kSortTile - 1) / kSortTile;
    PhaseScope ps(sim, NB_PHASE_TOPOLOGY, 6);
    NB_TRY(launch_after(k_gather_final, (n + 255) / 256, 256, 0, st, pos, t.keys[0], t.keys[1], t.vals[0],
                        t.vals[1], n, t.plan, t.spos, kMortonLevels, (const int32_t*)nullptr, (const int32_t*)nullptr));
    // this scan also clears the internal-node hash table for the emission
    NB_TRY(launch_after(k_positions_scan, ntiles, kPosThreads, 0, st, tv, t.spos, t.pos_nint, t.leaf_level,
                        t.leaf_count, t.counters, t.pos_status, ntiles, counts_only ? nullptr : t.hkeys, t.hash_cap,
                        nullptr, sim->d_err));
    if (counts_only) return cudaGetLastError();   // the node counts are in counters[TC_NINT], [TC_NLEAF]
    NB_TRY(launch_after(k_emit, nbk, kEmitBlock, 0, st, tv, t.pos_nint, t.int_level, t.int_first, t.int_code,
                        t.hkeys, t.hvals, hmask, t.int_mask, t.int_nint, t.int_pending, t.counters, t.popc_status,
                        ptiles));
    NB_TRY(launch_after(k_link, ib + nbk, kEmitBlock, 0, st, t.int_level, t.int_first, t.int_code, tv, icap,
                        t.counters + TC_NINT, ib, t.pos_nint, t.leaf_level, t.hkeys, t.hvals, hmask, t.int_parent,
                        t.leaf_parent, t.int_mask, t.int_nint, t.counters));
    NB_TRY(launch_after(k_popc_scan, ptiles, kPosThreads, 0, st, t.int_mask, icap, t.counters + TC_NINT,
                        t.int_block, t.counters, t.popc_status, ptiles, sim->d_err));
    NB_TRY(launch_after(k_place, ib + nbk, kEmitBlock, 0, st, t.int_level, t.int_code, t.int_parent, t.int_mask,
                        t.int_block, icap, t.counters + TC_NINT, ib, tv, t.leaf_level, t.leaf_count, t.leaf_parent,
                        t.spos, sim->prm.bounds_half, 1.0f, t.int_cell, t.cell_com, t.cell_mass, t.cell_count,
                        t.cell_meta, t.cell_lo, t.cell_hi, t.cell_code, rec));
    return cudaGetLastError();
}

// Capacity of the node arrays for a batched build: exact counts are measured
// once with a synchronising build and doubled (positions evolve).
cudaError_t tree_reserve_graph(nb_sim* sim, int n, size_t n_int, size_t n_cells) {
    const size_t nk = pad_up(std::max<size_t>((size_t)n, 1), kSortTile);
    NB_TRY(reserve_bodies(sim, nk));
    return reserve_nodes(sim, n_int, n_cells);
}

int tree_sort_tile() { return kSortTile; }

}  // namespace nb
