// nb_batch_kernels.cuh -- kernels of the batched form (included by nb_batch.cu).
//
// Many independent galaxies are stepped together, one launch per phase:
//  * Barnes-Hut members (n >= threshold) are stored first, contiguously.  Each
//    gets a tight bounding cube; a body's key is its galaxy slot (21 bits, the
//    top 7 octal levels) followed by a 42-bit code of its octants in its cube
//    (14 levels, sorted in Hilbert order), so ONE radix sort and ONE topology build make a forest whose
//    level-7 nodes are the galaxy roots.
//  * The mass pass adds traceless quadrupole moments (parallel-axis rule
//    bottom-up); a cell's centre of mass, walk record and quadrupole form one
//    64-byte record (nb_cellrec.cuh).  Traversal groups are
//    taken from the tree itself: runs of at most kGroupMax bodies of the
//    largest subtrees of at most kGroupCut bodies whose cell is at most 1/16
//    of the galaxy cube, the bodies in Hilbert order -- so a group is
//    spatially compact and its bounding box small.  A warp
//    takes groups from a device queue (two bodies per lane; one for groups of
//    at most 32 bodies, so that half-empty warps do no idle work), opens a
//    cell when the cell side exceeds theta times the distance from the cell's
//    centre of mass to the group's bounding box, and collects accepted cells
//    (monopole + quadrupole) and leaf buckets of at most leaf_size bodies
//    (summed body by body) in shared-memory lists that every lane then
//    evaluates for its bodies with the packed FP32x2 instructions; accepted
//    cells far from the group go into the group's local expansion instead.
//    This is a performance form whose parity is the force error against the
//    FP64 direct sum (<= 1e-3), not the reference's per-body opening rule.
//  * Direct-sum members are padded to multiples of 256 bodies; the warps of a
//    persistent kernel take (galaxy, target rows, source range) units from a
//    table through an atomic counter, each pair of bodies once, and a second
//    kernel folds the partials.
#pragma once

#include <type_traits>

#include "nb_morton.cuh"
#include "nb_cellrec.cuh"

namespace nb {

constexpr int kGWarps = 4;              // warps per traversal block
constexpr int kGroupMax = 64;           // bodies per traversal group (two per lane)
constexpr int kGroupCut = 512;          // most bodies of a cell that is cut into groups
constexpr int kGroupMinDepth = 4;       // such a cell lies >= 4 levels below its galaxy root
constexpr int kGroupFirstDepth = 7;     // groups of cells up to this depth are walked first
constexpr int kBoxChunk = 2048;         // bodies per block of the bounding-box pass (8 a thread)
constexpr int kGStack = 512;            // cells waiting to be opened, per warp (<= 32 pushed per step)
constexpr int kStackCellLimit = 1 << 27;   // a stack entry packs a first-child index below this with 4 bits
constexpr int kGMultiTop = kGStack - 155 - 32;   // stack height up to which a walk step takes several cells
constexpr int kGCells = 64;             // accepted-cell list, per warp
constexpr int kGBodies = 192;           // gathered leaf-bucket bodies, per warp
constexpr int kDirOnceMax = 8192;       // padded bodies up to which a direct member takes each pair once
// far-field defaults of the group traversal (rules in nb_batch.cu's nb_batch)
constexpr double kFarEta = 0.2;         // geometric rule: group half-diagonal / distance
constexpr double kFarAlpha = 1e-4;      // relative rule: truncation estimate / (|a|_min / G)
constexpr double kFarCap = 0.5;         // relative rule: largest half-diagonal / distance


// ---- per-body galaxy tables -------------------------------------------------
constexpr int kFillChunk = 8192;   // bodies per block of the table fill
// run = (first entry, entries, value, table): table 0 is the Barnes-Hut bodies'
// slot, table 1 the direct-sum bodies' galaxy.
__global__ void k_fill_tables(const int4* __restrict__ runs, int32_t* __restrict__ slot, int32_t* __restrict__ dgal) {
    const int4 r = runs[blockIdx.x];
    int32_t* out = r.w ? dgal : slot;
    for (int i = threadIdx.x; i < r.y; i += blockDim.x) out[r.x + i] = r.z;
}

// ---- whole-batch state transfer ----------------------------------------------
// The galaxies' bodies between the batch's arrays and one dense array in galaxy
// order, a run of at most kMoveChunk bodies a block: run = (first body in the
// arrays, first in the dense order, bodies, 0).  One copy each way then replaces
// one a galaxy, about 2 us each: reading 200 small galaxies back took 790 us.
constexpr int kMoveChunk = 2048;
template <bool GATHER>
__global__ void __launch_bounds__(256) k_move_state(const int4* __restrict__ runs, float4* __restrict__ state,
                                                    float4* __restrict__ dense) {
    const int4 r = runs[blockIdx.x];
    for (int i = threadIdx.x; i < r.z; i += blockDim.x) {
        if (GATHER) dense[r.y + i] = state[r.x + i];
        else state[r.x + i] = dense[r.y + i];
    }
}

// ---- bounding cube of each Barnes-Hut galaxy ------------------------------
// Min/max are exact and order-free, so chunks of kBoxChunk bodies reduce in
// parallel into per-galaxy words with atomics on an order-preserving integer
// image of the float (nb_morton.cuh).
//
// The first kernel of a batched step also clears the step's counters: the
// tree counters and the radix histograms (TC_NIN set to the bodies in the
// forest), the interaction count, the traversal group counters and the unit
// counters of the direct-sum launches.
__global__ void k_gal_box_init(unsigned* __restrict__ bits, int nslot, int32_t* __restrict__ counters,
                               int counter_words, int n_in, unsigned long long* __restrict__ interactions,
                               int* __restrict__ group_ctr, int* __restrict__ next_unit, int n_next) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 6 * nslot) bits[i] = (i % 6) < 3 ? 0xffffffffu : 0u;
    for (int j = i; j < counter_words; j += gridDim.x * blockDim.x) counters[j] = j == TC_NIN ? n_in : 0;
    if (i == 0) {
        *interactions = 0ull;
        group_ctr[0] = group_ctr[1] = group_ctr[2] = 0;
    }
    for (int j = i; j < n_next; j += gridDim.x * blockDim.x) next_unit[j] = 0;
}

__device__ __forceinline__ void box_flush(unsigned* bits, int slot, const float lo[3], const float hi[3]) {
    for (int a = 0; a < 3; ++a) {
        atomicMin(&bits[6 * slot + a], float_to_ordered(lo[a]));
        atomicMax(&bits[6 * slot + 3 + a], float_to_ordered(hi[a]));
    }
}

// block b reduces bodies [b*kBoxChunk, (b+1)*kBoxChunk) of the Barnes-Hut range.
// Latency-bound: eight dependent loads a thread instead of 32, four times the blocks.
__global__ void __launch_bounds__(256) k_gal_box_chunks(const float4* __restrict__ pos,
                                                        const int32_t* __restrict__ body_slot, int n, int nslot,
                                                        unsigned* __restrict__ bits) {
    const int base = blockIdx.x * kBoxChunk;
    const int end = min(n, base + kBoxChunk);
    int cur = -1;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int i = base + threadIdx.x; i < end; i += blockDim.x) {
        const int s = body_slot[i];
        if (s < 0 || s >= nslot) continue;
        if (s != cur) {
            if (cur >= 0) box_flush(bits, cur, lo, hi);
            cur = s;
            lo[0] = lo[1] = lo[2] = INFINITY;
            hi[0] = hi[1] = hi[2] = -INFINITY;
        }
        const float4 p = pos[i];
        lo[0] = fminf(lo[0], p.x); lo[1] = fminf(lo[1], p.y); lo[2] = fminf(lo[2], p.z);
        hi[0] = fmaxf(hi[0], p.x); hi[1] = fmaxf(hi[1], p.y); hi[2] = fmaxf(hi[2], p.z);
    }
    // a warp that ended in one galaxy reduces its bounds; a block that did adds one set of atomics
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ int sh_gal;
    __shared__ float sh_box[8][6];
    if (threadIdx.x == 0) sh_gal = cur;
    __syncthreads();
    const int c0 = sh_gal;
    const bool one = __syncthreads_and(cur == c0 || cur < 0) != 0;   // no body: neutral bounds
    const int w0 = __shfl_sync(0xffffffffu, cur, 0);
    if (__all_sync(0xffffffffu, cur == w0 || cur < 0)) {
        for (int a = 0; a < 3; ++a)
            for (int o = 16; o > 0; o >>= 1) {
                lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
                hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
            }
        if (lane == 0 && w0 >= 0 && !one) box_flush(bits, w0, lo, hi);
        if (lane == 0 && one)
            for (int a = 0; a < 3; ++a) {
                sh_box[warp][a] = lo[a];
                sh_box[warp][3 + a] = hi[a];
            }
    } else if (cur >= 0) {
        box_flush(bits, cur, lo, hi);
    }
    if (one) {   // block-uniform
        __syncthreads();
        if (threadIdx.x == 0 && c0 >= 0) {
            for (int w = 1; w < 8; ++w)
                for (int a = 0; a < 3; ++a) {
                    lo[a] = fminf(lo[a], sh_box[w][a]);
                    hi[a] = fmaxf(hi[a], sh_box[w][3 + a]);
                }
            box_flush(bits, c0, lo, hi);
        }
    }
}

// ---- bottom-up mass, centre of mass and quadrupole --------------------------
// Q_ij = sum m (3 y_i y_j - |y|^2 d_ij), y = offset from the node's centre of
// mass; a parent sums its children's Q plus m_c (3 d d - |d|^2 I), d = com_c - com.
// Leaf records are written by the placement (nb_cellrec.cuh); an internal
// node reads its children's records (contiguous) and writes its own whole.
// The children are read at once (eight predicated loads each, in registers:
// dynamically indexed arrays went through local memory): a batched step of one
// 1M-body galaxy went from 3.43 to 3.34 ms.
__device__ __forceinline__ void finish_moments(int c, int F, int nch, int first, int level, CellRec* rec) {
    float4 ccm[8], cq1[8], cq2[8];
    int cnt[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (j < nch) {
            const CellRec* r = rec + F + j;
            ccm[j] = load_published(&r->com);
            cnt[j] = load_published(&r->walk.y);
            cq1[j] = load_published(&r->q1);
            cq2[j] = load_published(&r->q2);
        }
    }
    float m = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
    int count = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (j < nch) {
            count += cnt[j];
            m += ccm[j].w;
            cx = fmaf(ccm[j].w, ccm[j].x, cx); cy = fmaf(ccm[j].w, ccm[j].y, cy); cz = fmaf(ccm[j].w, ccm[j].z, cz);
        }
    }
    const float im = m > 0.f ? 1.f / m : 0.f;
    cx *= im; cy *= im; cz *= im;
    float xx = 0.f, yy = 0.f, zz = 0.f, xy = 0.f, xz = 0.f, yz = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (j < nch) {
            const float mc = ccm[j].w;
            const float dx = ccm[j].x - cx, dy = ccm[j].y - cy, dz = ccm[j].z - cz, r2 = dx * dx + dy * dy + dz * dz;
            xx += cq1[j].x + mc * (3.f * dx * dx - r2);
            yy += cq1[j].y + mc * (3.f * dy * dy - r2);
            zz += cq1[j].z + mc * (3.f * dz * dz - r2);
            xy += cq2[j].x + mc * 3.f * dx * dy;
            xz += cq2[j].y + mc * 3.f * dx * dz;
            yz += cq2[j].z + mc * 3.f * dy * dz;
        }
    }
    CellRec* r = rec + c;
    __stcg(&r->com, make_float4(cx, cy, cz, m));
    __stcg(&r->walk, walk_record(F, count, first, BK_INTERNAL, nch, level));
    __stcg(&r->q1, make_float4(xx, yy, zz, 0.f));
    __stcg(&r->q2, make_float4(xy, xz, yz, 0.f));
}

// One thread per internal node whose children are all leaves; the last child
// of a node to finish finishes the node (acquire-release counter per node).
// The bound is the chain of round trips from the deepest node to its root: a
// node's own words are read while the arrival counter is on the way, and a
// node with one internal child needs no counter (its other children are
// leaves, complete since the placement).  In large states it is the nodes in
// flight: 128 registers give four blocks an SM where 137 gave three (a step of 180
// galaxies of 8192 to 65,536 bodies 8.98 -> 8.85 ms, of 16 x 65,536 2.63 -> 2.61; 96
// registers spill: 8.95).  Eight lanes a node, at 40 registers, took 9.02.
__global__ void __launch_bounds__(128, 4) k_batch_moments(
    int int_cap, const int32_t* __restrict__ counters, const int32_t* __restrict__ int_parent,
    const int32_t* __restrict__ int_nint, int32_t* __restrict__ int_pending, const int32_t* __restrict__ int_cell,
    const int32_t* __restrict__ int_block, const uint32_t* __restrict__ int_mask,
    const int32_t* __restrict__ int_first, const int32_t* __restrict__ int_level, CellRec* __restrict__ rec,
    int cell_cap, int* __restrict__ err) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (!tree_fits(counters, int_cap, cell_cap)) return;   // held step: no moments
    const int ni = min(counters[TC_NINT], int_cap);
    if (k >= ni || int_nint[k] != 0) return;
    int c = int_cell[k], F = 1 + int_block[k], nch = __popc(int_mask[k]), first = int_first[k], level = int_level[k];
    int parent = k > 0 ? int_parent[k] : -1;
    for (int guard = 0; guard < 64; ++guard) {
        if (c < 0 || c >= cell_cap || F + nch > cell_cap) record_error(err, DEV_TREE_OVERFLOW);   // corrupt node
        else finish_moments(c, F, nch, first, level, rec);
        const int p = parent;
        if (k == 0 || p < 0 || p >= ni) return;
        const int nint = int_nint[p];
        c = int_cell[p];
        F = 1 + int_block[p];
        nch = __popc(int_mask[p]);
        first = int_first[p];
        level = int_level[p];
        parent = p > 0 ? int_parent[p] : -1;
        if (nint > 1) {
            const int old = atomic_add_acq_rel(&int_pending[p], 1);   // publishes this node, sees its siblings
            if (old != nint - 1) return;
        }
        k = p;
    }
}

// Root cell of each galaxy: the level-7 internal node starting at the
// galaxy's first sorted position.
__global__ void k_batch_roots(const int32_t* __restrict__ slot_start, int nslot, const uint64_t* __restrict__ keys,
                              const int32_t* __restrict__ int_base, const int32_t* __restrict__ int_cell,
                              const int32_t* __restrict__ counters, int int_cap, int cell_cap,
                              int32_t* __restrict__ root, int32_t* __restrict__ err) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nslot) return;
    if (!tree_fits(counters, int_cap, cell_cap)) return;   // held step: no walk
    const int s = slot_start[g];
    int prev = -1;
    if (s > 0) {
        const uint64_t x = keys[s - 1] ^ keys[s];
        prev = x == 0 ? kBatchDepth : (__clzll((long long)x) - (64 - 3 * kBatchDepth)) / 3;
    }
    const int k = int_base[s] + (kSlotLevels - (prev + 1));
    if (prev + 1 > kSlotLevels || k < 0 || k >= min(counters[TC_NINT], int_cap)) {
        root[g] = -1;
        record_error(err, DEV_TREE_OVERFLOW);
        return;
    }
    root[g] = int_cell[k];
}

// ---- traversal groups from the tree --------------------------------------------
// One thread per internal node at or below the galaxy roots.  A cell of at most
// kGroupCut bodies that lies deep enough (groupable) is cut into runs of at most
// kGroupMax bodies of nearly equal length, which are compact because bodies are
// sorted along the Hilbert curve; groupable children that follow one another on
// the curve are cut together when their parent is deep enough.  A node that is
// not groupable handles its groupable children, emits a body that sits high in
// the tree on its own and cuts a larger depth-cap bucket; its other children are
// handled by their own threads.  Every body lands in exactly one group: a run of
// the first groupable cell on its path from the galaxy root, or its leaf.
// Before, a group was a whole cell of at most 64 bodies or consecutive siblings
// packed to 64 in Morton order, which left 33% of the traversal's slots empty at
// 1M bodies (14% now): a step 3.34 -> 2.95 ms there, 1.25 -> 1.14 ms at 300,000.
// The group boxes are no larger, and the force error falls (2.6e-4 -> 2.5e-4 and,
// with the relative far field, 5.4e-4 -> 4.9e-4 at 1M).
// Groups of the cells up to kGroupFirstDepth levels below their galaxy's root go
// to the front of the list and are walked first, the others fill it from the
// back: the longest walks are those of wide groups next to a dense region, and
// one that starts last holds the whole launch.
struct GroupList {
    int4* list;
    int cap;
    int* ctr;   // [0] groups at the front, [1] next group to walk, [2] groups at the back
};
constexpr int kGroupCounters = 3;

__device__ __forceinline__ void emit_group(int first, int count, bool front, const int32_t* sorder,
                                           const int32_t* body_slot, int nbodies, const GroupList& g, int* err) {
    if (count <= 0) return;
    if (first < 0 || first + count > nbodies) {
        record_error(err, DEV_TREE_OVERFLOW);
        return;
    }
    const int idx = atomicAdd(&g.ctr[front ? 0 : 2], 1);
    if (idx >= g.cap) {   // groups are disjoint and not empty: at most one a body
        record_error(err, DEV_TREE_OVERFLOW);
        return;
    }
    g.list[front ? idx : g.cap - 1 - idx] = make_int4(body_slot[sorder[first]], first, count, 0);
}

// A cell can be cut into groups when it lies at least kGroupMinDepth levels below
// its galaxy's root (side <= cube / 16): a few bodies spread over a large,
// sparse cell would give one group a box the size of the galaxy and a list of
// ~10^5 entries (a tail that held one warp for milliseconds); such cells are
// split further instead.  For the same reason a cell at that depth is cut only
// when it makes one group, and twice as many bodies are allowed every two levels
// deeper, up to kGroupCut (doubling at every level left long walks at the end:
// 1.29 ms a step at 300,000 bodies; up to 512 everywhere 1.67 ms).
__device__ __forceinline__ bool groupable(int level, int count) {
    const int depth = level - kSlotLevels - kGroupMinDepth;
    return depth >= 0 && count <= min(kGroupCut, kGroupMax << min(depth / 2, 8));
}

__device__ __forceinline__ void emit_runs(int first, int count, bool front, const int32_t* sorder,
                                          const int32_t* body_slot, int nbodies, const GroupList& g, int* err) {
    const int runs = (count + kGroupMax - 1) / kGroupMax;
    for (int r = 0; r < runs; ++r) {
        const int o = (int)((long long)count * r / runs), e = (int)((long long)count * (r + 1) / runs);
        emit_group(first + o, e - o, front, sorder, body_slot, nbodies, g, err);
    }
}

__global__ void __launch_bounds__(256) k_batch_groups(int int_cap, const int32_t* __restrict__ counters,
                                                      const int32_t* __restrict__ int_cell,
                                                      const CellRec* __restrict__ rec,
                                                      const int32_t* __restrict__ sorder,
                                                      const int32_t* __restrict__ body_slot, int n_cells, int nbodies,
                                                      GroupList groups, int* __restrict__ err) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    // a held step emits no groups, so the traversal after it has no work
    if (!tree_fits(counters, int_cap, n_cells)) return;
    if (k >= min(counters[TC_NINT], int_cap)) return;
    const int c = int_cell[k];
    if (c < 0 || c >= n_cells) {
        record_error(err, DEV_TREE_OVERFLOW);
        return;
    }
    const int4 wr = rec[c].walk;
    const int level = wr.w >> 8;
    const int cnt = wr.y;
    if (level < kSlotLevels) return;
    if (groupable(level, cnt)) return;   // its parent cuts it
    const int F = wr.x, nch = (wr.w >> 4) & 15;
    if (F < 1 || nch > 8 || F + nch > n_cells) {
        record_error(err, DEV_TREE_OVERFLOW);
        return;
    }
    // children are cut together only below a cell small enough itself
    const bool pack = level >= kSlotLevels + kGroupMinDepth;
    const bool front = level < kSlotLevels + kGroupFirstDepth;   // the children's level is one more
    int first[8], count[8], kind[8];
    bool can[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        first[j] = 0x7fffffff;
        count[j] = kind[j] = 0;
        can[j] = false;
        if (j < nch) {
            const int4 cw = rec[F + j].walk;
            kind[j] = cw.w & 15;
            count[j] = cw.y;
            first[j] = cw.z;
            can[j] = groupable(cw.w >> 8, cw.y);
        }
    }
    int run_first = -1, run_cnt = 0, last = -1;
    for (int it = 0; it < nch; ++it) {   // the children along the curve
        int cf = 0x7fffffff, cc = 0, ck = 0;
        bool cg = false;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (first[j] > last && first[j] < cf) {
                cf = first[j];
                cc = count[j];
                ck = kind[j];
                cg = can[j];
            }
        last = cf;
        if (cg && pack) {
            if (run_first < 0) run_first = cf;
            run_cnt += cc;
            continue;
        }
        if (run_cnt) emit_runs(run_first, run_cnt, front, sorder, body_slot, nbodies, groups, err);
        run_first = -1;
        run_cnt = 0;
        // a groupable child of a cell high in the tree, a body high in the tree or a
        // larger depth-cap bucket; another internal child cuts its own children
        if (cg || ck != BK_INTERNAL) emit_runs(cf, cc, front, sorder, body_slot, nbodies, groups, err);
    }
    if (run_cnt) emit_runs(run_first, run_cnt, front, sorder, body_slot, nbodies, groups, err);
}

// Interactions of one target (negated coordinates duplicated in both halves
// of n*) with TWO accepted cells at once (their values paired in the float2
// operands): monopole with the force law plus the Newtonian quadrupole term,
//   a += w x - Q x / r^5 + 5/2 (x.Q.x) x / r^7,  x = com - p,
// w the force law's (softened) monopole factor.  The list holds -Q (the q*
// arguments), which saves a negation per pair.  Under the reference law 1/r
// comes from the law's own reciprocal square root,
//   1/r = (r^2 + S) / sqrt(r^2 (r^2 + S)^2),
// one multiply instead of a second reciprocal square root.
template <int LAW>
__device__ __forceinline__ void cell_pair_accel(float2 cx, float2 cy, float2 cz, float2 cm, float2 qxx, float2 qyy,
                                                float2 qzz, float2 qxy, float2 qxz, float2 qyz, float2 nx, float2 ny,
                                                float2 nz, float2 S2, float2 T2, float2& ax, float2& ay, float2& az) {
    const float2 dx = __fadd2_rn(cx, nx);
    const float2 dy = __fadd2_rn(cy, ny);
    const float2 dz = __fadd2_rn(cz, nz);
    float2 r2 = __fmul2_rn(dx, dx);
    r2 = __ffma2_rn(dy, dy, r2);
    r2 = __ffma2_rn(dz, dz, r2);
    float2 w, ir;
    if (LAW == NB_LAW_REFERENCE) {
        const float2 s = __fadd2_rn(r2, S2);
        const float2 t = __ffma2_rn(__fmul2_rn(r2, s), s, T2);
        const float2 rt = make_float2(rsqrt_approx(t.x), rsqrt_approx(t.y));
        w = __fmul2_rn(cm, rt);
        ir = __fmul2_rn(rt, s);
    } else {
        const float2 q = __fadd2_rn(r2, S2);
        const float2 inv = make_float2(rsqrt_approx(q.x), rsqrt_approx(q.y));
        w = __fmul2_rn(__fmul2_rn(cm, inv), __fmul2_rn(inv, inv));
        ir = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
    }
    const float2 ir2 = __fmul2_rn(ir, ir);
    const float2 ir5 = __fmul2_rn(__fmul2_rn(ir2, ir), ir2);
    // q = -Q x, xqx = -x.Q.x
    const float2 qx = __ffma2_rn(qxx, dx, __ffma2_rn(qxy, dy, __fmul2_rn(qxz, dz)));
    const float2 qy = __ffma2_rn(qxy, dx, __ffma2_rn(qyy, dy, __fmul2_rn(qyz, dz)));
    const float2 qz = __ffma2_rn(qxz, dx, __ffma2_rn(qyz, dy, __fmul2_rn(qzz, dz)));
    const float2 xqx = __ffma2_rn(dx, qx, __ffma2_rn(dy, qy, __fmul2_rn(dz, qz)));
    const float2 c7 = __fmul2_rn(ir5, __fmul2_rn(ir2, make_float2(-2.5f, -2.5f)));
    const float2 wc = __ffma2_rn(xqx, c7, w);
    ax = __ffma2_rn(wc, dx, __ffma2_rn(ir5, qx, ax));
    ay = __ffma2_rn(wc, dy, __ffma2_rn(ir5, qy, ay));
    az = __ffma2_rn(wc, dz, __ffma2_rn(ir5, qz, az));
}

// Shared-memory lists hold their entries in pairs, each value of the two
// entries side by side, so that one 16-byte load yields two FP32x2 operands:
// a body pair is (x x' y y')(z z' m m'), a cell pair (x x' y y')(z z' m m')
// then -Q: (Qxx Qxx' Qyy Qyy')(Qzz Qzz' Qxy Qxy')(Qxz Qxz' Qyz Qyz'), negated.
constexpr float kFarAway = 1e18f;   // position of the zero-mass cell that pads an odd list

__device__ __forceinline__ void put_body(float4 (*lst)[2], int j, float4 b) {
    float* f = reinterpret_cast<float*>(lst[j >> 1]);
    const int h = j & 1;
    f[h] = b.x; f[2 + h] = b.y; f[4 + h] = b.z; f[6 + h] = b.w;
}

__device__ __forceinline__ void put_cell(float4 (*lst)[5], int j, float4 cm, float4 q1, float4 q2) {
    float* f = reinterpret_cast<float*>(lst[j >> 1]);
    const int h = j & 1;
    f[h] = cm.x; f[2 + h] = cm.y; f[4 + h] = cm.z; f[6 + h] = cm.w;
    f[8 + h] = -q1.x; f[10 + h] = -q1.y; f[12 + h] = -q1.z; f[14 + h] = -q2.x;
    f[16 + h] = -q2.y; f[18 + h] = -q2.z;
}

// Far field of a group: accepted cells that are far from the group compared
// with its size (group half-diagonal < eta * distance from the box centre X)
// act through a local expansion at X instead of once per body:
//   a(X + y) = A + J y + 1/2 H(y, y) + 1/6 T(y, y, y),
// A the cell's full acceleration at X (force law + quadrupole), J the first
// derivative of its Newtonian monopole + quadrupole field, H and T the second
// and third derivatives of the monopole field (with d = COM - X, r = |d|,
// s = d.Q.d):
//   J_ij   = m (3 d_i d_j / r^5 - delta_ij / r^3)
//          + Q_ij / r^5 - 5 ((Qd)_i d_j + (Qd)_j d_i) / r^7 - 5/2 s delta_ij / r^7 + 35/2 s d_i d_j / r^9,
//   H_ijk  = m (15 d_i d_j d_k / r^7 - 3 (delta_ik d_j + delta_jk d_i + delta_ij d_k) / r^5),
//   T_ijkl = m (105 d_i d_j d_k d_l / r^9 - 15 (delta_ij d_k d_l + 5 more pairings) / r^7
//               + 3 (delta_ij delta_kl + delta_ik delta_jl + delta_il delta_jk) / r^5)
// (the quadrupole part of J is minus the derivative, with respect to d, of
// the quadrupole acceleration -Q d / r^5 + 5/2 s d / r^7).  Each is a
// derivative tensor of a harmonic potential, so every trace vanishes and only
// the independent components are summed: J 5 (zz = -xx - yy), H 7 (xzz, yzz,
// zzz from the traces), T 9 (xxzz, yyzz, zzzz, xyzz, xzzz, yzzz from the
// traces).  The truncation error of a cell's term falls as (size / distance)^4.
constexpr int kFarTerms = 24;   // A (3), J xx yy xy xz yz (5), H (7), T (9)
struct FarField {
    float v[kFarTerms];
};

// Adds one cell's terms to a lane's partial sums in shared memory, four terms a
// 16-byte word (term 4 k + c is component c of f[k * stride]): a quarter of the
// loads and stores of single terms.
template <int LAW>
__device__ __forceinline__ void far_add(float4* f, int stride, const float4 cm, const float4 q1, const float4 q2,
                                        float Xx, float Xy, float Xz, float S) {
    const float dx = cm.x - Xx, dy = cm.y - Xy, dz = cm.z - Xz;
    const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    const float m = cm.w;
    float w;
    if (LAW == NB_LAW_REFERENCE) {
        const float s = r2 + S;
        w = m * rsqrt_approx(fmaf(r2 * s, s, kTiny));
    } else {
        const float inv = rsqrt_approx(r2 + S);
        w = m * inv * (inv * inv);
    }
    const float ir = rsqrt_approx(r2), ir2 = ir * ir, ir3 = ir2 * ir, ir5 = ir3 * ir2, ir7 = ir5 * ir2;
    // quadrupole term at X (Q traceless: q1 = Qxx Qyy Qzz, q2 = Qxy Qxz Qyz)
    const float qx = fmaf(q1.x, dx, fmaf(q2.x, dy, q2.y * dz));
    const float qy = fmaf(q2.x, dx, fmaf(q1.y, dy, q2.z * dz));
    const float qz = fmaf(q2.y, dx, fmaf(q2.z, dy, q1.z * dz));
    const float sq = fmaf(dx, qx, fmaf(dy, qy, dz * qz));   // d.Q.d
    const float c7 = 2.5f * sq * ir7;
    float4 t;
    auto T = [&](int k, float x) {
        switch (k & 3) {   // k is a constant
            case 0: t = f[(k >> 2) * stride]; t.x += x; break;
            case 1: t.y += x; break;
            case 2: t.z += x; break;
            default: t.w += x; f[(k >> 2) * stride] = t;
        }
    };
    T(0, fmaf(w + c7, dx, -qx * ir5));
    T(1, fmaf(w + c7, dy, -qy * ir5));
    T(2, fmaf(w + c7, dz, -qz * ir5));
    const float m3 = 3.f * m * ir5, m1 = m * ir3;
    const float t5 = 5.f * ir7, g9 = 17.5f * sq * ir7 * ir2, dg = m1 + c7;   // c7 = 5/2 s / r^7
    T(3, fmaf(m3 * dx, dx, -dg) + fmaf(q1.x, ir5, dx * fmaf(g9, dx, -2.f * t5 * qx)));   // J xx
    T(4, fmaf(m3 * dy, dy, -dg) + fmaf(q1.y, ir5, dy * fmaf(g9, dy, -2.f * t5 * qy)));   // J yy
    T(5, fmaf(m3 * dx + g9 * dx, dy, fmaf(q2.x, ir5, -t5 * fmaf(qx, dy, qy * dx))));     // J xy
    T(6, fmaf(m3 * dx + g9 * dx, dz, fmaf(q2.y, ir5, -t5 * fmaf(qx, dz, qz * dx))));     // J xz
    T(7, fmaf(m3 * dy + g9 * dy, dz, fmaf(q2.z, ir5, -t5 * fmaf(qy, dz, qz * dy))));     // J yz
    const float m15 = 15.f * m * ir7;
    const float tx = m15 * dx, ty = m15 * dy;
    T(8, dx * fmaf(tx, dx, -3.f * m3));    // H xxx = 15 m dx^3 / r^7 - 9 m dx / r^5
    T(9, dy * fmaf(ty, dy, -3.f * m3));    // H yyy
    T(10, dy * fmaf(tx, dx, -m3));         // H xxy
    T(11, dz * fmaf(tx, dx, -m3));         // H xxz
    T(12, dx * fmaf(ty, dy, -m3));         // H xyy
    T(13, dz * fmaf(ty, dy, -m3));         // H yyz
    T(14, tx * dy * dz);                   // H xyz
    const float a9 = 105.f * m * ir7 * ir2;           // 105 m / r^9
    const float x2 = dx * dx, y2 = dy * dy;
    const float ax2 = a9 * x2, ay2 = a9 * y2;
    T(15, fmaf(x2, ax2 - 6.f * m15, 3.f * m3));          // T xxxx
    T(16, fmaf(y2, ay2 - 6.f * m15, 3.f * m3));          // T yyyy
    T(17, fmaf(ax2, y2, fmaf(-m15, x2 + y2, m3)));        // T xxyy
    T(18, dx * dy * (ax2 - 3.f * m15));                  // T xxxy
    T(19, dx * dy * (ay2 - 3.f * m15));                  // T xyyy
    T(20, dx * dz * (ax2 - 3.f * m15));                  // T xxxz
    T(21, dx * dz * (ay2 - m15));                        // T xyyz
    T(22, dy * dz * (ax2 - m15));                        // T xxyz
    T(23, dy * dz * (ay2 - 3.f * m15));                  // T yyyz
}

// A + J y + 1/2 H(y, y) + 1/6 T(y, y, y) at offset y from the expansion centre.
__device__ __forceinline__ void far_eval(const FarField& f, float x, float y, float z, float& ax, float& ay,
                                         float& az) {
    const float* v = f.v;
    const float Jxx = v[3], Jyy = v[4], Jxy = v[5], Jxz = v[6], Jyz = v[7], Jzz = -Jxx - Jyy;
    const float Hxxx = v[8], Hyyy = v[9], Hxxy = v[10], Hxxz = v[11], Hxyy = v[12], Hyyz = v[13], Hxyz = v[14];
    const float Hxzz = -Hxxx - Hxyy, Hyzz = -Hxxy - Hyyy, Hzzz = -Hxxz - Hyyz;
    const float Txxxx = v[15], Tyyyy = v[16], Txxyy = v[17], Txxxy = v[18], Txyyy = v[19], Txxxz = v[20],
                Txyyz = v[21], Txxyz = v[22], Tyyyz = v[23];
    const float Txxzz = -Txxxx - Txxyy, Tyyzz = -Txxyy - Tyyyy, Tzzzz = -Txxzz - Tyyzz;
    const float Txyzz = -Txxxy - Txyyy, Txzzz = -Txxxz - Txyyz, Tyzzz = -Txxyz - Tyyyz;
    const float xx = x * x, yy = y * y, zz = z * z, xy = x * y, xz = x * z, yz = y * z;
    const float x3 = xx * x, y3 = yy * y, z3 = zz * z;
    const float x2y = xx * y, x2z = xx * z, xy2 = x * yy, y2z = yy * z, xz2 = x * zz, yz2 = y * zz, xyz = xy * z;
    constexpr float s6 = 1.f / 6.f;
    ax = v[0] + Jxx * x + Jxy * y + Jxz * z + 0.5f * (Hxxx * xx + Hxyy * yy + Hxzz * zz) + Hxxy * xy + Hxxz * xz +
         Hxyz * yz + s6 * (Txxxx * x3 + Txyyy * y3 + Txzzz * z3) +
         0.5f * (Txxxy * x2y + Txxxz * x2z + Txxyy * xy2 + Txxzz * xz2 + Txyyz * y2z + Txyzz * yz2) + Txxyz * xyz;
    ay = v[1] + Jxy * x + Jyy * y + Jyz * z + 0.5f * (Hxxy * xx + Hyyy * yy + Hyzz * zz) + Hxyy * xy + Hxyz * xz +
         Hyyz * yz + s6 * (Txxxy * x3 + Tyyyy * y3 + Tyzzz * z3) +
         0.5f * (Txxyy * x2y + Txxyz * x2z + Txyyy * xy2 + Txyzz * xz2 + Tyyyz * y2z + Tyyzz * yz2) + Txyyz * xyz;
    az = v[2] + Jxz * x + Jyz * y + Jzz * z + 0.5f * (Hxxz * xx + Hyyz * yy + Hzzz * zz) + Hxyz * xy + Hxzz * xz +
         Hyzz * yz + s6 * (Txxxz * x3 + Tyyyz * y3 + Tzzzz * z3) +
         0.5f * (Txxyz * x2y + Txxzz * x2z + Txyyz * xy2 + Txzzz * xz2 + Tyyzz * y2z + Tyzzz * yz2) + Txyzz * xyz;
}

// Persistent: each warp takes groups from the queue until it is empty.
// Bound by instruction issue (62% of the cycles, five warps a scheduler, their
// stalls mostly the fixed latency of dependent instructions): a group of 52
// bodies meets 368 cells and 1917 bodies in 90 walk steps at 1,048,576 bodies, a
// third to the bodies' evaluation and nearly half to the steps.  Four body pairs
// an iteration, four far-field terms a shared-memory word, exact powers of two
// for ldexpf and the gather below: 2.93 -> 2.76 ms a step there, 16 galaxies of
// 65,536 2.78 -> 2.63, 200 of 2048 to 8192 1.64 -> 1.57.
template <int LAW>
__global__ void __launch_bounds__(kGWarps * 32, 5) k_group_traverse(
    GroupList groups,
    const float4* __restrict__ spos, const int32_t* __restrict__ sorder, const CellRec* __restrict__ rec,
    const float4* __restrict__ gal_box, const int32_t* __restrict__ gal_root, int nslot, int n_cells, int nbodies,
    int max_pops, int leaf_size, float theta2, float S, float G, float far2, float far_rel, float far_cap2,
    float far_min_r2,
    const unsigned* __restrict__ mmax, float4* __restrict__ acc,
    unsigned long long* __restrict__ inter, int* __restrict__ err) {
    __shared__ int stk[kGWarps][kGStack];
    __shared__ float4 lcl[kGWarps][kGCells / 2][5];
    __shared__ float4 lbd[kGWarps][kGBodies / 2][2];
    __shared__ float4 ffs[kGWarps][kFarTerms / 4][32];   // far-field partial sums, one column per lane
    __shared__ int rfst[kGWarps][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const float2 S2 = make_float2(S, S);
    const float tiny = self_pair_tiny(mmax);   // a leaf's bodies include the target itself
    const float2 T2 = make_float2(tiny, tiny);
    unsigned long long total = 0;
    for (;;) {
    int gi = 0;
    if (lane == 0) gi = atomicAdd(&groups.ctr[1], 1);
    gi = __shfl_sync(0xffffffffu, gi, 0);
    const int nfront = min(groups.ctr[0], groups.cap);   // read again for each group: two registers less
    if (gi >= nfront + min(groups.ctr[2], groups.cap - nfront)) break;
    const int4 grp = groups.list[gi < nfront ? gi : groups.cap - 1 - (gi - nfront)];   // (slot, first sorted position, count, 0)
    if (grp.x < 0 || grp.x >= nslot || grp.y < 0 || grp.z < 1 || grp.z > kGroupMax || grp.y + grp.z > nbodies) {
        if (lane == 0) record_error(err, DEV_TREE_OVERFLOW);
        continue;
    }
    const bool v0 = lane < grp.z, v1 = lane + 32 < grp.z;
    const bool dual = grp.z > 32;   // warp-uniform: groups of at most 32 bodies evaluate one body per lane
    const int s0 = grp.y + (v0 ? lane : 0), s1 = grp.y + (v1 ? lane + 32 : 0);
    const float4 p0 = spos[s0], p1 = spos[s1];
    float bl[3], bh[3];
    {
        const float a0[3] = {p0.x, p0.y, p0.z}, a1[3] = {p1.x, p1.y, p1.z};
        for (int a = 0; a < 3; ++a) {
            bl[a] = fminf(v0 ? a0[a] : INFINITY, v1 ? a1[a] : INFINITY);
            bh[a] = fmaxf(v0 ? a0[a] : -INFINITY, v1 ? a1[a] : -INFINITY);
            for (int o = 16; o > 0; o >>= 1) {
                bl[a] = fminf(bl[a], __shfl_xor_sync(0xffffffffu, bl[a], o));
                bh[a] = fmaxf(bh[a], __shfl_xor_sync(0xffffffffu, bh[a], o));
            }
        }
    }
    const float4 gb = gal_box[grp.x];
    // expansion centre of the group's far field and its half-diagonal squared
    const float Xx = 0.5f * (bl[0] + bh[0]), Xy = 0.5f * (bl[1] + bh[1]), Xz = 0.5f * (bl[2] + bh[2]);
    const float rg2 = 0.25f * ((bh[0] - bl[0]) * (bh[0] - bl[0]) + (bh[1] - bl[1]) * (bh[1] - bl[1]) +
                               (bh[2] - bl[2]) * (bh[2] - bl[2]));
    // relative far-field rule: the group's smallest |a| / G of the previous
    // evaluation (none yet: 0, the geometric rule decides)
    float far_thr = 0.f;
    if (far_rel > 0.f) {
        float a2 = INFINITY;
        if (v0) {
            const float4 a = acc[sorder[s0]];
            a2 = fmaf(a.z, a.z, fmaf(a.y, a.y, a.x * a.x));
        }
        if (v1) {
            const float4 a = acc[sorder[s1]];
            a2 = fminf(a2, fmaf(a.z, a.z, fmaf(a.y, a.y, a.x * a.x)));
        }
        for (int o = 16; o > 0; o >>= 1) a2 = fminf(a2, __shfl_xor_sync(0xffffffffu, a2, o));
        if (a2 > 0.f && a2 < INFINITY) far_thr = far_rel * sqrtf(a2);
    }
    const bool use_far = far2 > 0.f || far_rel > 0.f;
    for (int k = 0; k < kFarTerms / 4; ++k) ffs[w][k][lane] = make_float4(0.f, 0.f, 0.f, 0.f);   // this lane's share of the far field
    // negated target coordinates, duplicated: the pair partner is the other list entry
    const float2 n0x = make_float2(-p0.x, -p0.x), n0y = make_float2(-p0.y, -p0.y), n0z = make_float2(-p0.z, -p0.z);
    const float2 n1x = make_float2(-p1.x, -p1.x), n1y = make_float2(-p1.y, -p1.y), n1z = make_float2(-p1.z, -p1.z);
    const float2 z2 = make_float2(0.f, 0.f);
    float2 a0x = z2, a0y = z2, a0z = z2, a1x = z2, a1y = z2, a1z = z2;   // (even entries, odd entries)
    float s0x = 0.f, s0y = 0.f, s0z = 0.f, c0x = 0.f, c0y = 0.f, c0z = 0.f;
    float s1x = 0.f, s1y = 0.f, s1z = 0.f, c1x = 0.f, c1y = 0.f, c1z = 0.f;
    unsigned cnt = 0;
    const unsigned nv = (v0 ? 1u : 0u) + (v1 ? 1u : 0u);
    int nst = 0, ncl = 0, nbd = 0, pops = 0;
    bool bad = false;

    auto fold = [&]() {
        kahan_add(s0x, c0x, a0x.x + a0x.y); kahan_add(s0y, c0y, a0y.x + a0y.y); kahan_add(s0z, c0z, a0z.x + a0z.y);
        kahan_add(s1x, c1x, a1x.x + a1x.y); kahan_add(s1y, c1y, a1y.x + a1y.y); kahan_add(s1z, c1z, a1z.x + a1z.y);
        a0x = a0y = a0z = a1x = a1y = a1z = z2;
    };
    auto flush_cells = [&]() {
        if (ncl & 1) {   // pad with a zero-mass, zero-moment cell far away: adds exactly zero
            if (lane == 0)
                put_cell(lcl[w], ncl, make_float4(kFarAway, kFarAway, kFarAway, 0.f), make_float4(0.f, 0.f, 0.f, 0.f),
                         make_float4(0.f, 0.f, 0.f, 0.f));
        }
        __syncwarp();
        auto cell_loop = [&](auto both) {
            for (int k = 0; k < (ncl + 1) >> 1; ++k) {
                const float4 e0 = lcl[w][k][0], e1 = lcl[w][k][1], e2 = lcl[w][k][2], e3 = lcl[w][k][3],
                             e4 = lcl[w][k][4];
                const float2 cx = make_float2(e0.x, e0.y), cy = make_float2(e0.z, e0.w), cz = make_float2(e1.x, e1.y);
                const float2 cm = make_float2(e1.z, e1.w), qxx = make_float2(e2.x, e2.y), qyy = make_float2(e2.z, e2.w);
                const float2 qzz = make_float2(e3.x, e3.y), qxy = make_float2(e3.z, e3.w), qxz = make_float2(e4.x, e4.y);
                const float2 qyz = make_float2(e4.z, e4.w);
                cell_pair_accel<LAW>(cx, cy, cz, cm, qxx, qyy, qzz, qxy, qxz, qyz, n0x, n0y, n0z, S2, T2, a0x, a0y,
                                     a0z);
                if (decltype(both)::value)
                    cell_pair_accel<LAW>(cx, cy, cz, cm, qxx, qyy, qzz, qxy, qxz, qyz, n1x, n1y, n1z, S2, T2, a1x, a1y,
                                         a1z);
            }
        };
        if (dual) cell_loop(std::true_type{}); else cell_loop(std::false_type{});
        cnt += nv * ncl;
        ncl = 0;
        fold();
        __syncwarp();
    };
    auto flush_bodies = [&]() {
        if (nbd & 1) {   // pad with a zero-mass body: adds exactly zero
            if (lane == 0) put_body(lbd[w], nbd, make_float4(0.f, 0.f, 0.f, 0.f));
        }
        __syncwarp();
        const int np = (nbd + 1) >> 1;
        auto body_loop = [&](auto both) {
            int k = 0;
#pragma unroll 1
            for (; k + 4 <= np; k += 4) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float4 e0 = lbd[w][k + u][0], e1 = lbd[w][k + u][1];
                    const float2 bx = make_float2(e0.x, e0.y), by = make_float2(e0.z, e0.w);
                    const float2 bz = make_float2(e1.x, e1.y), bm = make_float2(e1.z, e1.w);
                    interact_x2<LAW>(bx, by, bz, bm, n0x, n0y, n0z, S2, T2, a0x, a0y, a0z);
                    if (decltype(both)::value)
                        interact_x2<LAW>(bx, by, bz, bm, n1x, n1y, n1z, S2, T2, a1x, a1y, a1z);
                }
            }
            for (; k < np; ++k) {
                const float4 e0 = lbd[w][k][0], e1 = lbd[w][k][1];
                const float2 bx = make_float2(e0.x, e0.y), by = make_float2(e0.z, e0.w);
                const float2 bz = make_float2(e1.x, e1.y), bm = make_float2(e1.z, e1.w);
                interact_x2<LAW>(bx, by, bz, bm, n0x, n0y, n0z, S2, T2, a0x, a0y, a0z);
                if (decltype(both)::value) interact_x2<LAW>(bx, by, bz, bm, n1x, n1y, n1z, S2, T2, a1x, a1y, a1z);
            }
        };
        if (dual) body_loop(std::true_type{}); else body_loop(std::false_type{});
        cnt += nv * nbd;
        nbd = 0;
        fold();
        __syncwarp();
    };
    // Appends the bodies of this step's accepted leaf ranges (lane l: first,
    // count; count 0 for lanes without one) to the body list, all lanes
    // copying, 32 bodies at a time, evaluating the list whenever it fills.  A
    // body's range is the last that starts at or before it: the starts of a
    // window as a bit mask (a binary search in the ranges' ends cost five
    // dependent reads a body; this took 3% off the batched step).  The list is
    // filled to its last place, so that its evaluation, four pairs at a time,
    // has no rest but at the walk's end: flushing at the last whole window instead
    // took all of that back.
    auto gather_ranges = [&](int first, int count) {
        int incl = count;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const int tot = __shfl_sync(0xffffffffu, incl, 31), start = incl - count;
        const uint32_t some = __ballot_sync(0xffffffffu, count > 0);
        __syncwarp();
        if (count > 0) rfst[w][__popc(some & lt)] = first - start;
        __syncwarp();
        int before = -1;   // the last range that starts before the window
        for (int done = 0, take; done < tot; done += take) {
            if (nbd == kGBodies) flush_bodies();
            take = min(min(32, kGBodies - nbd), tot - done);
            const unsigned at = (unsigned)(start - done);
            const uint32_t starts = __reduce_or_sync(0xffffffffu, count > 0 && at < (unsigned)take ? 1u << at : 0u);
            if (lane < take)
                put_body(lbd[w], nbd + lane, spos[rfst[w][before + __popc(starts & ((2u << lane) - 1u))] + done + lane]);
            before += __popc(starts);
            nbd += take;
        }
        __syncwarp();
    };

    const int root = gal_root[grp.x];
    if (root < 1 || root >= n_cells) {
        bad = true;
    } else {
        const int4 rw = __ldg(&rec[root].walk);
        const int rF = rw.x, rn = (rw.w >> 4) & 15;
        if ((rw.w & 15) != BK_INTERNAL || rF < 1 || rn < 1 || rn > 8 || rF + rn > n_cells || rF >= kStackCellLimit) {
            bad = true;
        } else {
            if (lane == 0) stk[w][0] = (rF << 4) | rn;
            nst = 1;
        }
    }
    __syncwarp();
    while (nst > 0 && !bad) {
        if (++pops > max_pops) { bad = true; break; }
        // Take up to 8 opened cells from the top of the stack, as many as have
        // at most 32 children together; lane j tests the j-th of those children.
        // Above kGMultiTop waiting cells a step takes one cell (a depth-first
        // walk leaving at most 7 cells per level, 7 * 21 + 8 in all), so the
        // stack stays below kGMultiTop + 31 + 155 < kGStack.
        const int cap = nst <= kGMultiTop ? 8 : 1;
        int pF = 0, pn = 0;
        if (lane < cap && lane < nst) {   // a stack entry is an opened cell's (first child << 4 | children)
            const int e = stk[w][nst - 1 - lane];
            pF = e >> 4;
            pn = e & 15;
        }
        int incl = pn;   // inclusive prefix of the child counts over lanes 0..7
        for (int o = 1; o < 8; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const uint32_t take = __ballot_sync(0xffffffffu, lane < cap && lane < nst && incl <= 32);
        const int P = __popc(take);   // >= 1: one cell has at most 8 children
        const int T = __shfl_sync(0xffffffffu, incl, P - 1);
        __syncwarp();
        nst -= P;
        // source cell of this lane's child: the last taken cell starting at or
        // before it (every opened cell has at least one child, so the starts differ)
        const uint32_t starts = __reduce_or_sync(0xffffffffu, lane < P ? 1u << (incl - pn) : 0u);
        const int q = __popc(starts & ((2u << lane) - 1u)) - 1;
        const int qF = __shfl_sync(0xffffffffu, pF, q & 7);
        const int qx = __shfl_sync(0xffffffffu, incl - pn, q & 7);
        bool a_cell = false, a_range = false, a_push = false, a_bad = false;
        float4 ccm = make_float4(0.f, 0.f, 0.f, 0.f);
        int first = 0, count = 0, ch = 0, cF = 0, cn = 0;
        if (lane < T) {
            ch = qF + (lane - qx);
            ccm = __ldg(&rec[ch].com);
            const int4 wr = __ldg(&rec[ch].walk);
            const int kind = wr.w & 15;
            count = wr.y;
            first = wr.z;
            cF = wr.x;
            cn = (wr.w >> 4) & 15;
            // The group form of the reference's rule side / r < theta: r is bounded
            // below for every body of the group by the distance from the centre of
            // mass to the group's bounding box.
            const float side = gb.w * __int_as_float((127 + kSlotLevels - (wr.w >> 8)) << 23);   // box size / 2^level
            float d2 = 0.f;
            const float cc[3] = {ccm.x, ccm.y, ccm.z};
            for (int a = 0; a < 3; ++a) {
                const float d = fmaxf(0.f, fmaxf(bl[a] - cc[a], cc[a] - bh[a]));
                d2 = fmaf(d, d, d2);
            }
            const bool accept = side * side < theta2 * d2;
            a_cell = accept && count > 2 && kind == BK_INTERNAL;
            a_range = !a_cell && (count <= leaf_size || kind != BK_INTERNAL);
            a_push = !a_cell && !a_range;
            if (a_cell && use_far) {
                const float ex = ccm.x - Xx, ey = ccm.y - Xy, ez = ccm.z - Xz;
                const float r2X = fmaf(ez, ez, fmaf(ey, ey, ex * ex));
                bool far;
                if (far_thr > 0.f) {   // m / r^2 (r_g / r)^4 < alpha |a|_min / G, r_g / r < cap
                    const float q = rg2 / r2X;
                    far = rg2 < far_cap2 * r2X && ccm.w * q * q < far_thr * r2X;
                } else {
                    far = rg2 < far2 * r2X;
                }
                if (far && r2X > far_min_r2) {   // far: into the group's local expansion
                    far_add<LAW>(&ffs[w][0][lane], 32, ccm, __ldg(&rec[ch].q1), __ldg(&rec[ch].q2), Xx, Xy, Xz, S);
                    cnt += (unsigned)grp.z;
                    a_cell = false;   // accepted, not listed
                }
            }
            // node data outside the body range would be a corrupt tree: report, never dereference
            if (a_range && (first < 0 || count < 0 || first + count > nbodies)) a_range = false, a_bad = true;
            if (a_push && (cF < 1 || cn < 1 || cn > 8 || cF + cn > n_cells || cF >= kStackCellLimit))
                a_push = false, a_bad = true;
        }
        if (__any_sync(0xffffffffu, a_bad)) { bad = true; break; }
        const uint32_t bc = __ballot_sync(0xffffffffu, a_cell);
        if (bc) {
            if (ncl + __popc(bc) > kGCells) flush_cells();
            if (a_cell) {
                const int idx = ncl + __popc(bc & lt);
                put_cell(lcl[w], idx, ccm, __ldg(&rec[ch].q1), __ldg(&rec[ch].q2));
            }
            ncl += __popc(bc);
        }
        const uint32_t br = __ballot_sync(0xffffffffu, a_range);
        if (br) gather_ranges(a_range ? first : 0, a_range ? count : 0);
        const uint32_t bp = __ballot_sync(0xffffffffu, a_push);
        if (bp) {
            if (nst + __popc(bp) > kGStack) { bad = true; break; }
            if (a_push) stk[w][nst + __popc(bp & lt)] = (cF << 4) | cn;
            nst += __popc(bp);
        }
        __syncwarp();
    }
    if (!bad) {
        flush_cells();
        flush_bodies();
    }
    fold();
    // the group's far field: sum the lanes' partial expansions, evaluate at each body
    if (use_far) {
        FarField ff;
#pragma unroll
        for (int k = 0; k < kFarTerms; ++k) {
            const float4 t = ffs[w][k >> 2][lane];
            float x = (k & 3) == 0 ? t.x : (k & 3) == 1 ? t.y : (k & 3) == 2 ? t.z : t.w;
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            ff.v[k] = x;
        }
        float fx, fy, fz;
        far_eval(ff, p0.x - Xx, p0.y - Xy, p0.z - Xz, fx, fy, fz);
        kahan_add(s0x, c0x, fx); kahan_add(s0y, c0y, fy); kahan_add(s0z, c0z, fz);
        far_eval(ff, p1.x - Xx, p1.y - Xy, p1.z - Xz, fx, fy, fz);
        kahan_add(s1x, c1x, fx); kahan_add(s1y, c1y, fy); kahan_add(s1z, c1z, fz);
    }
    if (bad && lane == 0) record_error(err, DEV_STACK_OVERFLOW);
    if (v0) acc[sorder[s0]] = make_float4(G * (s0x - c0x), G * (s0y - c0y), G * (s0z - c0z), 0.f);
    if (v1) acc[sorder[s1]] = make_float4(G * (s1x - c1x), G * (s1y - c1y), G * (s1z - c1z), 0.f);
    total += cnt;
    }
    for (int o = 16; o > 0; o >>= 1) total += __shfl_down_sync(0xffffffffu, total, o);
    if (lane == 0 && total) atomicAdd(inter, total);
}

// ---- batched direct sum --------------------------------------------------------
// A unit is a row of 32 * IPT target bodies, IPT a lane in registers (packed
// FP32x2), against a run of 32-source chunks: (first target body, first source
// body, chunks | chunks evaluated from the target side only << 16, entry of the
// target partials); unit_src is the entry of body 0 among the row's source
// partials, or, with APART, the distance of the compensations from the targets' sums.  Sources behind the row are evaluated once for both bodies, 17
// FP32 operations for two interactions instead of 26: lane l takes source
// (l + r) mod 32 at step r, and the sources' sums travel with them by shuffle
// (as in k_direct_pairs, here within one warp).  The row's own bodies, and all
// sources of a member of more than kDirOnceMax padded bodies (whose source
// partials would grow with its square), are evaluated from the target side
// (direct_chunk).  Such a member's few partials keep sum and compensation apart
// (APART): rounded to one word they added 2% to the force error at 9000 and 16,000 bodies.
// (Where each pair is taken once, the many partials of a body carry less: the error
// is 4% below that of the target side with both parts.)
//
// Bound by the FP32 pipe.  Warps share nothing, so that no barrier waits for
// the slowest; the next chunk and the next unit are fetched while the current
// chunk is evaluated.  GB300, 200 members of 256-4096 bodies: force
// kernel 387 -> 235 us and the fold 8 -> 34 us (ncu, cold caches; it now reads a
// partial per row and body), ten steps and a read 4.76 -> 2.83 ms; FMA pipe 63% busy, the rest
// is the shuffles and reads that four targets a lane carry (eight: 268 us a
// step, but small members then fill fewer rows).
constexpr int kDirWarps = 8;   // most warps per block
template <int LAW, int IPT, bool APART>
__global__ void __launch_bounds__(kDirWarps * 32, IPT == 4 ? 2 : 1) k_batch_direct(
    const float4* __restrict__ pos, const int4* __restrict__ units, const int32_t* __restrict__ unit_src, int nunits,
    int* __restrict__ next_unit, float S, const unsigned* __restrict__ mmax, float4* __restrict__ part) {
    __shared__ float4 src[kDirWarps][2][kDirChunk];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float tiny = self_pair_tiny(mmax);
    const float2 S2 = make_float2(S, S), T2 = make_float2(tiny, tiny);
    constexpr int P = IPT / 2;
    int u = 0;
    if (lane == 0) u = atomicAdd(next_unit, 1);
    u = __shfl_sync(0xffffffffu, u, 0);
    while (u < nunits) {
        const int4 un = units[u];
        const int src0 = unit_src[u], chunks = un.z & 0xffff, own = un.z >> 16;
        int after = 0;
        if (lane == 0) after = atomicAdd(next_unit, 1);
        float2 nx[P], ny[P], nz[P], mi[P];
        float sum[3 * IPT], comp[3 * IPT];
#pragma unroll
        for (int q = 0; q < P; ++q) {
            const float4 a = pos[un.x + (2 * q) * 32 + lane], b = pos[un.x + (2 * q + 1) * 32 + lane];
            nx[q] = make_float2(-a.x, -b.x);
            ny[q] = make_float2(-a.y, -b.y);
            nz[q] = make_float2(-a.z, -b.z);
            mi[q] = make_float2(a.w, b.w);
        }
#pragma unroll
        for (int k = 0; k < 3 * IPT; ++k) sum[k] = comp[k] = 0.f;
        float4 cur = pos[un.y + lane];
        for (int c = 0; c < chunks; ++c) {
            float4* buf = src[warp][c & 1];
            buf[lane] = cur;
            __syncwarp();   // also: every lane is done with the chunk that this buffer held
            if (c + 1 < chunks) cur = pos[un.y + (c + 1) * kDirChunk + lane];
            float3 f;
            if (APART || c < own) {
                direct_chunk<LAW, IPT, false>(buf, lane, nx, ny, nz, mi, S2, T2, sum, comp, f);
            } else {
                direct_chunk<LAW, IPT, true>(buf, lane, nx, ny, nz, mi, S2, T2, sum, comp, f);
                part[(long long)src0 + un.y + c * kDirChunk + lane] = make_float4(f.x, f.y, f.z, 0.f);
            }
        }
        if (APART) {
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                const size_t at = (size_t)un.w + k * 32 + lane;
                part[at] = make_float4(sum[3 * k], sum[3 * k + 1], sum[3 * k + 2], 0.f);
                part[at + src0] = make_float4(comp[3 * k], comp[3 * k + 1], comp[3 * k + 2], 0.f);
            }
        } else {
#pragma unroll
            for (int k = 0; k < IPT; ++k)
                part[(size_t)un.w + k * 32 + lane] =
                    make_float4(sum[3 * k] - comp[3 * k], sum[3 * k + 1] - comp[3 * k + 1], sum[3 * k + 2] - comp[3 * k + 2], 0.f);
        }
        u = __shfl_sync(0xffffffffu, after, 0);
        __syncwarp();   // the next unit's first chunk may take the buffer read last
    }
}

// A direct-sum member's partials: [splits][n_pad] for its bodies as targets
// (only the first ones of a row that its sources fill), then, where each pair
// is taken once, for each row one entry per body behind it, else the targets'
// compensations, [splits][n_pad] again.
struct DirGal {
    int off, n_pad, row, split;   // first body, padded bodies, bodies a row, source bodies a unit
    int base, splits, once, sources;   // first entry, splits, each pair once?, source bodies (to a whole chunk)
};

// Folds the partials of direct-sum body i (global index begin + i) into acc, in
// a fixed order: a block's warps share 32 bodies (of one row).  With eight
// neighbouring threads a body instead, whose reads are a row apart, the fold of 200
// members of 256-4096 bodies took 44 us instead of 34, a step 294 instead of 283.
__global__ void __launch_bounds__(32 * kFoldWarps) k_batch_direct_reduce(const int32_t* __restrict__ body_dgal,
                                                                         const DirGal* __restrict__ dgal, int begin,
                                                                         float G, const float4* __restrict__ part,
                                                                         float4* __restrict__ acc) {
    __shared__ float sums[kFoldWarps][6][32];
    const int i = blockIdx.x * 32 + (threadIdx.x & 31), j = threadIdx.x >> 5;
    const int g = body_dgal[i];
    float ax = 0.f, ay = 0.f, az = 0.f, kx = 0.f, ky = 0.f, kz = 0.f;
    if (g >= 0) {   // not a padding body
        const DirGal d = dgal[g];
        const int local = begin + i - d.off, row = local / d.row;
        auto add = [&](const float4 p) {
            kahan_add(ax, kx, p.x);
            kahan_add(ay, ky, p.y);
            kahan_add(az, kz, p.z);
        };
        const int behind = d.sources - (d.once ? row * d.row : 0);
        const int used = (behind + d.split - 1) / d.split;
#pragma unroll 4
        for (int s = j; s < used; s += kFoldWarps) add(part[(size_t)d.base + (size_t)s * d.n_pad + local]);
        if (d.once) {
            const float4* src = part + (size_t)d.base + (size_t)d.splits * d.n_pad;
#pragma unroll 4
            for (int r = j; r < row; r += kFoldWarps)
                add(src[(size_t)r * d.n_pad - (size_t)d.row * r * (r + 1) / 2 + (local - (r + 1) * d.row)]);
        } else {
            const float4* low = part + (size_t)d.base + (size_t)d.splits * d.n_pad + local;
            float qx = 0.f, qy = 0.f, qz = 0.f;
#pragma unroll 4
            for (int s = j; s < used; s += kFoldWarps) {
                const float4 c = low[(size_t)s * d.n_pad];
                qx += c.x; qy += c.y; qz += c.z;
            }
            kx += qx; ky += qy; kz += qz;
        }
    }
    const float3 f = add_warps(sums, ax, ay, az, kx, ky, kz).rounded();
    if (g >= 0 && j == 0) acc[begin + i] = make_float4(G * f.x, G * f.y, G * f.z, 0.f);
}

}  // namespace nb
