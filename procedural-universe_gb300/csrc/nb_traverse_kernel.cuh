// nb_traverse_kernel.cuh -- the K6 traversal kernel (included by nb_traverse.cu).
//
// A warp walks the tree for 64 consecutive bodies of the key order, two per
// lane (lane l holds bodies base + l and base + 32 + l).  Every body still
// makes exactly the decisions of the reference's recursion; what changes is
// where they are made:
//   * Each popped cell's children are first classified for the whole group
//     at once, one lane per child, from the group's bounding box: if even the
//     nearest point of the box is beyond the cell's accept distance, every
//     body of the group accepts the cell (its float r^2 exceeds the accept
//     threshold); if even the farthest corner is inside the reject distance,
//     every body opens it.  Both bounds carry a 1e-5 relative margin, far
//     above the few-ulp rounding of the float distances, so a group verdict
//     never differs from a body's own.
//   * Cells every body accepts, and one-body leaves, go to one shared-memory
//     list (with the lane masks of the bodies that reached them, less a leaf's
//     own body) that is evaluated densely for both bodies of every lane with
//     the packed FP32x2 instructions; cells every body opens are pushed without
//     per-body work.
//   * Only the remaining ("ambiguous") cells and depth-cap buckets are decided
//     body by body, as the reference does, with the accept / reject
//     thresholds and the exactly rounded ratio inside the 2e-5 band.
// A stack entry carries one lane mask per body slot: the bodies that opened
// that cell.
//
// Bound by instruction issue and the walk's dependency chains.  Sources of both
// kinds share one list, whose entries are evaluated four at a time so that their
// chains interleave: 3.79 -> 3.60 ms at 1,048,576 bodies (bodies in Morton
// order).  Where the groups are too few to fill the GPU, K warps of a block
// share one.
#pragma once

namespace nb {

constexpr int kMultiTop = kStack - 176 - 32;   // stack height up to which a step takes several entries
static_assert(kMultiTop > 0, "stack too small for multi-entry steps");
constexpr int kRun = 4;           // list entries evaluated together
constexpr int kList = 64;   // sources waiting for evaluation, per warp (a step adds at most 32)
constexpr int kListRoom = 6 * kTravBodies * 4 / 16;   // room for a warp's sums when a group is shared
static_assert(kListRoom >= kList, "the list fits");

// The interactions of a lane's two bodies with one source (its coordinates
// broadcast in both halves); m carries the source mass per body, zero where
// that body takes no interaction.
template <int LAW>
__device__ __forceinline__ void pair_accel_x2(float2 dx, float2 dy, float2 dz, float2 r2, float2 m, float2 S2,
                                              float2& ax, float2& ay, float2& az) {
    float2 w;
    if (LAW == NB_LAW_REFERENCE) {
        const float2 s = __fadd2_rn(r2, S2);
        const float2 t = __ffma2_rn(__fmul2_rn(r2, s), s, make_float2(kTravTiny, kTravTiny));
        w = __fmul2_rn(m, make_float2(rsqrt_approx(t.x), rsqrt_approx(t.y)));
    } else {
        const float2 q = __fadd2_rn(r2, S2);
        const float2 inv = make_float2(rsqrt_approx(q.x), rsqrt_approx(q.y));
        w = __fmul2_rn(__fmul2_rn(m, inv), __fmul2_rn(inv, inv));
    }
    ax = __ffma2_rn(w, dx, ax);
    ay = __ffma2_rn(w, dy, ay);
    az = __ffma2_rn(w, dz, az);
}

// A source at c acting on the lane's two bodies (negated coordinates n*).
template <int LAW>
__device__ __forceinline__ void source_accel_x2(const float4 c, float2 m, float2 nx, float2 ny, float2 nz, float2 S2,
                                                float2& ax, float2& ay, float2& az) {
    const float2 dx = __fadd2_rn(make_float2(c.x, c.x), nx);
    const float2 dy = __fadd2_rn(make_float2(c.y, c.y), ny);
    const float2 dz = __fadd2_rn(make_float2(c.z, c.z), nz);
    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
    pair_accel_x2<LAW>(dx, dy, dz, r2, m, S2, ax, ay, az);
}

// Pairwise force of each body of an opened depth-cap bucket on body p.
template <int LAW>
__device__ __forceinline__ void bucket_accel(const float4* __restrict__ spos, int first, int count, int n, int self,
                                             const float4 p, float S, float& ax, float& ay, float& az,
                                             unsigned& cnt) {
    const int qe = min(first + count, n);
    for (int q = max(first, 0); q < qe; ++q) {
        if (q == self) continue;
        const float4 bq = spos[q];
        const float dx = bq.x - p.x, dy = bq.y - p.y, dz = bq.z - p.z;
        pair_accel<LAW>(dx, dy, dz, fmaf(dz, dz, fmaf(dy, dy, dx * dx)), bq.w, S, ax, ay, az);
        ++cnt;
    }
}

// Waiting entries at which a shared group's warps part: sooner, the parts are uneven,
// later, the steps made alike are more.  A step by 6, 12 and 24: 4000 bodies 222, 195
// and 227 us, 10,000 282, 262 and 304, 40,000 376, 365 and 372 (1000: 153, 161 and 161;
// 60,000: 469, 482 and 490).
constexpr int kSplitAt = 12;
enum : int { CL_NONE = -1, CL_SOURCE = 0, CL_OPEN = 2, CL_DECIDE = 3, CL_EMPTY = 4 };

// BLOCKS: blocks an SM is to hold, which sets the registers (4: 126; 0, the
// compiler's own choice: 96 and five blocks; asked for five outright it does
// 1.5% worse at 1,048,576 bodies).
template <int LAW, int K, int BLOCKS>
__global__ void __launch_bounds__(kTravBlock, BLOCKS) k_traverse(const float4* __restrict__ spos,
                                                         const int32_t* __restrict__ sorder, int n,
                                                         const float4* __restrict__ cell_com,
                                                         const int4* __restrict__ cell_meta,
                                                         const float4* __restrict__ cell_lo, int n_cells,
                                                         int max_pops, float theta_f, float S, float G,
                                                         float4* __restrict__ acc,
                                                         unsigned long long* __restrict__ inter,
                                                         int* __restrict__ err) {
    // 12-byte entries (child range, lanes of body slot 0, of slot 1): the smaller the
    // shared-memory footprint, the more of the SM's L1 is left for the node reads
    struct StackEntry { int range, lanes0, lanes1; };
    __shared__ StackEntry stk[kTravWarps][kStack];
    __shared__ float4 kid_cm[kTravWarps][32];
    __shared__ int4 kid_mt[kTravWarps][32];
    __shared__ unsigned kid_ch[kTravWarps][32];
    __shared__ float4 ls_src[kTravWarps][K > 1 ? kListRoom : kList];
    __shared__ uint2 ls_mask[kTravWarps][kList];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, part = K > 1 ? w % K : 0;
    const uint32_t lt = (1u << lane) - 1u, bit = 1u << lane;
    const int base = (blockIdx.x * kTravWarps + w) / K * kTravBodies;
    const int s0 = base + lane, s1 = base + 32 + lane;
    const bool v0 = s0 < n, v1 = s1 < n;
    if (K == 1 && base >= n) return;   // a warp past the last body
    const float4 p0 = v0 ? spos[s0] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 p1 = v1 ? spos[s1] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float2 nx = make_float2(-p0.x, -p1.x), ny = make_float2(-p0.y, -p1.y), nz = make_float2(-p0.z, -p1.z);
    const float2 S2 = make_float2(S, S), z2 = make_float2(0.f, 0.f);
    const unsigned cell_lim = min((unsigned)n_cells, 1u << kRangeBits);
    // the group's bounding box (valid bodies)
    float glo[3], ghi[3];
    {
        const float a0[3] = {p0.x, p0.y, p0.z}, a1[3] = {p1.x, p1.y, p1.z};
        for (int a = 0; a < 3; ++a) {
            glo[a] = fminf(v0 ? a0[a] : INFINITY, v1 ? a1[a] : INFINITY);
            ghi[a] = fmaxf(v0 ? a0[a] : -INFINITY, v1 ? a1[a] : -INFINITY);
            for (int o = 16; o > 0; o >>= 1) {
                glo[a] = fminf(glo[a], __shfl_xor_sync(0xffffffffu, glo[a], o));
                ghi[a] = fmaxf(ghi[a], __shfl_xor_sync(0xffffffffu, ghi[a], o));
            }
        }
    }
    float2 sx = z2, sy = z2, sz = z2, cx = z2, cy = z2, cz = z2;   // totals and negated compensations
    float2 tx = z2, ty = z2, tz = z2;
    unsigned cnt = 0;
    // The list fills from both ends: sources that every valid body of the warp
    // takes from the front, evaluated without masks; the others from the back,
    // with their masks.
    int top = 0, pops = 0, nf = 0, np = 0;
    const unsigned vm0 = __ballot_sync(0xffffffffu, v0), vm1 = __ballot_sync(0xffffffffu, v1);
    bool bad = false;

    auto fold = [&]() {
        kahan_add_x2(sx, cx, tx); kahan_add_x2(sy, cy, ty); kahan_add_x2(sz, cz, tz);
        tx = ty = tz = z2;
    };
    auto take_full = [&](int k) {
        const float4 c = ls_src[w][k];
        source_accel_x2<LAW>(c, make_float2(c.w, c.w), nx, ny, nz, S2, tx, ty, tz);
    };
    auto take_part = [&](int k) {
        const float4 c = ls_src[w][k];
        const uint2 mk = ls_mask[w][k];
        const float2 m = make_float2((mk.x & bit) ? c.w : 0.f, (mk.y & bit) ? c.w : 0.f);
        source_accel_x2<LAW>(c, m, nx, ny, nz, S2, tx, ty, tz);
    };
    // The list's length bounds the terms summed in plain FP32 before a fold.
    auto flush = [&]() {
        __syncwarp();
        int k = 0;
#pragma unroll 1
        for (; k + kRun <= nf; k += kRun) {   // independent chains interleave
#pragma unroll
            for (int u = 0; u < kRun; ++u) take_full(k + u);
            if (K > 1 && (k & 31) == 32 - kRun) fold();   // a small state's forces come from few terms
        }
#pragma unroll 1
        for (; k < nf; ++k) take_full(k);
        fold();
        const int back = kList - np;
        k = 0;
#pragma unroll 1
        for (; k + kRun <= np; k += kRun) {
#pragma unroll
            for (int u = 0; u < kRun; ++u) take_part(back + k + u);
            if (K > 1 && (k & 31) == 32 - kRun) fold();
        }
#pragma unroll 1
        for (; k < np; ++k) take_part(back + k);
        nf = np = 0;
        fold();
        __syncwarp();
    };

    // A walk step takes up to 8 entries from the top of the stack, as many as
    // have at most 32 children together; lane j handles the j-th of those
    // children (cell ch), reached by the bodies of its entry's masks (cm0, cm1).
    // The first step is the root, reached by every valid body.
    // With K > 1 the K warps of a group make the first steps alike, of which
    // only part 0 keeps the sources; once kSplitAt entries wait, each takes
    // every K-th of them and walks on alone.
    bool shared = K > 1, mine = part == 0;
    int T = (K > 1 && base >= n) ? 0 : 1;   // a group past the last body: nothing to walk
    unsigned ch = 0;
    unsigned cm0 = vm0, cm1 = vm1;
    // A shared group's warps are few (the GPU is not full): the children of the
    // next step are loaded before the list is evaluated, which then hides them: 4000
    // bodies 147 -> 130 us, 30,000 203 -> 184, 60,000 431 -> 396.  With a warp a group
    // other warps do that, and the fuller list is worth more (2^20: 3.06 ms, so 3.15).
    float4 ccm = make_float4(0.f, 0.f, 0.f, 0.f);
    int4 cmt = make_int4(0, 0, 0, 0);
    auto fetch = [&]() {
        cmt.w = 0;
        if ((int)lane < T) {
            ccm = __ldg(&cell_com[ch]);
            cmt = __ldg(&cell_meta[ch]);
        }
    };
    if (K > 1) fetch();
    while (T > 0) {
        // ---- classify the children for the whole group, one lane per child ----
        int cls = CL_NONE;
        if (K == 1) {
            ccm = make_float4(0.f, 0.f, 0.f, 0.f);
            cmt = make_int4(0, 0, 0, 0);
            fetch();
        }
        if ((int)lane < T) {
            kid_cm[w][lane] = ccm;
            kid_mt[w][lane] = cmt;
            kid_ch[w][lane] = ch;
            const int kind = cmt.w & 15;
            if (kind == TK_SINGLE) {
                cls = CL_SOURCE;
            } else if (kind != TK_INTERNAL) {
                cls = CL_DECIDE;   // depth-cap bucket: body by body
            } else {
                const float c[3] = {ccm.x, ccm.y, ccm.z};
                float dmin2 = 0.f, dmax2 = 0.f;
                for (int a = 0; a < 3; ++a) {
                    // nearest and farthest point of the group's box along this axis
                    const float dl = glo[a] - c[a], dh = ghi[a] - c[a];
                    const float dn = fmaxf(0.f, fmaxf(dl, -dh));
                    const float df = fmaxf(fabsf(dh), fabsf(dl));
                    dmin2 = fmaf(dn, dn, dmin2);
                    dmax2 = fmaf(df, df, dmax2);
                }
                const float thr_acc = __int_as_float(cmt.y), thr_rej = __int_as_float(cmt.z);
                if (dmin2 * (1.f - 1e-5f) > thr_acc) cls = ccm.w != 0.f ? CL_SOURCE : CL_EMPTY;
                else if (dmax2 * (1.f + 1e-5f) < thr_rej) cls = CL_OPEN;
                else cls = CL_DECIDE;
            }
        }
        __syncwarp();
        const unsigned bO = __ballot_sync(0xffffffffu, cls == CL_OPEN);
        const unsigned bD = __ballot_sync(0xffffffffu, cls == CL_DECIDE);
        // sources: one-body leaves (every body that reached them takes the pair, not the
        // body itself) and cells every body accepts (the monopole, for every body that
        // reached them)
        if (mine) {
            bool full = cm0 == vm0 && cm1 == vm1;
            unsigned m0 = cm0, m1 = cm1;
            if ((cmt.w & 15) == TK_SINGLE) {
                const unsigned slot = (unsigned)(cmt.x - base);
                if (slot < (unsigned)kTravBodies) {   // one of the group's own bodies
                    if (slot < 32u) m0 &= ~(1u << slot); else m1 &= ~(1u << (slot & 31u));
                    full = false;
                }
            }
            const unsigned bF = __ballot_sync(0xffffffffu, cls == CL_SOURCE && full);
            const unsigned bP = __ballot_sync(0xffffffffu, cls == CL_SOURCE && !full);
            if (bF | bP) {
                if (K == 1 && nf + np + __popc(bF | bP) > kList) flush();
                if (cls == CL_SOURCE) {
                    if (full) {
                        ls_src[w][nf + __popc(bF & lt)] = ccm;
                    } else {
                        const int k = kList - 1 - (np + __popc(bP & lt));
                        ls_src[w][k] = ccm;
                        ls_mask[w][k] = make_uint2(m0, m1);
                    }
                    cnt += __popc(m0) + __popc(m1);
                }
                nf += __popc(bF);
                np += __popc(bP);
            }
        }
        // cells every body opens
        if (bO) {
            bool ok = true;
            if (cls == CL_OPEN) {
                const unsigned cf = (unsigned)cmt.x, cn = ((unsigned)cmt.w >> 4) & 15u;
                ok = cf < cell_lim && cn - 1u < 8u && cf + cn <= cell_lim;
                if (ok && top + __popc(bO) <= kStack)
                    stk[w][top + __popc(bO & lt)] = StackEntry{(int)(cf | (cn << kRangeBits)), (int)cm0, (int)cm1};
            }
            if (!__all_sync(0xffffffffu, ok) || top + __popc(bO) > kStack) bad = true;
            top += __popc(bO);
        }
        // the rest: each body decides, as the reference's recursion does
        // Two ambiguous children per iteration: their arithmetic is independent,
        // so the two dependency chains interleave; the stack receives the first
        // child's entry before the second's, as one child per iteration would.
        auto decide = [&](int j, unsigned pm0, unsigned pm1, bool& open0, bool& open1) {
            const float4 cm = kid_cm[w][j];
            const int4 mt = kid_mt[w][j];
            const bool a0 = (pm0 & bit) != 0u, a1 = (pm1 & bit) != 0u;
            // the reference's float distance: dv = p - COM, r2 = (dvx^2 + dvy^2) + dvz^2; d = COM - p
            // = -dv exactly (rounding is symmetric).  The reference rounds every operation; the
            // compiler contracts packed products and sums (never the scalar intrinsics), so r2 may
            // differ in its last bit.  In some 2e8 decisions one body takes a cell that the
            // reference opens: 13 of 191,159,588 interactions at 155,648 bodies.
            const float2 dx = __fadd2_rn(make_float2(cm.x, cm.x), nx);
            const float2 dy = __fadd2_rn(make_float2(cm.y, cm.y), ny);
            const float2 dz = __fadd2_rn(make_float2(cm.z, cm.z), nz);
            const float2 r2 = __fadd2_rn(__fadd2_rn(__fmul2_rn(dx, dx), __fmul2_rn(dy, dy)), __fmul2_rn(dz, dz));
            const float thr_acc = __int_as_float(mt.y), thr_rej = __int_as_float(mt.z);
            bool acc0 = r2.x > thr_acc, acc1 = r2.y > thr_acc;
            const bool band0 = a0 && !acc0 && !(r2.x < thr_rej), band1 = a1 && !acc1 && !(r2.y < thr_rej);
            if (band0 || band1) {
                const float side = __ldg(&cell_lo[kid_ch[w][j]]).w;
                if (band0) acc0 = __fdiv_rn(side, __fsqrt_rn(r2.x)) < theta_f;
                if (band1) acc1 = __fdiv_rn(side, __fsqrt_rn(r2.y)) < theta_f;
            }
            acc0 = acc0 && a0;
            acc1 = acc1 && a1;
            // a body that does not take the cell adds an exact zero (zero mass, finite factor)
            const float mass = mine ? cm.w : 0.f;
            pair_accel_x2<LAW>(dx, dy, dz, r2, make_float2(acc0 ? mass : 0.f, acc1 ? mass : 0.f), S2, tx, ty, tz);
            if (mass != 0.f) cnt += (acc0 ? 1u : 0u) + (acc1 ? 1u : 0u);
            const int kind = mt.w & 15;
            if (kind == TK_INTERNAL) {
                open0 = a0 && !acc0;
                open1 = a1 && !acc1;
            } else {
                // opened depth-cap bucket: each of its bodies except the body itself
                const int bc = mt.w >> 8;
                if (mine && a0 && !acc0) bucket_accel<LAW>(spos, mt.x, bc, n, s0, p0, S, tx.x, ty.x, tz.x, cnt);
                if (mine && a1 && !acc1) bucket_accel<LAW>(spos, mt.x, bc, n, s1, p1, S, tx.y, ty.y, tz.y, cnt);
                open0 = open1 = false;
            }
        };
        auto push = [&](int j, bool open0, bool open1) {
            const unsigned b0 = __ballot_sync(0xffffffffu, open0), b1 = __ballot_sync(0xffffffffu, open1);
            if (b0 | b1) {
                const int4 mt = kid_mt[w][j];
                const unsigned cf = (unsigned)mt.x, cn = ((unsigned)mt.w >> 4) & 15u;
                if (top < kStack && cf < cell_lim && cn - 1u < 8u && cf + cn <= cell_lim) {
                    if (lane == 0) stk[w][top] = StackEntry{(int)(cf | (cn << kRangeBits)), (int)b0, (int)b1};
                    ++top;
                } else {
                    bad = true;
                }
            }
        };
        for (unsigned rem = bD; rem && !bad;) {
            const int j = __ffs(rem) - 1;
            rem &= rem - 1u;
            const bool two = rem != 0u;   // warp-uniform
            const int k = two ? __ffs(rem) - 1 : j;
            if (two) rem &= rem - 1u;
            const unsigned pj0 = __shfl_sync(0xffffffffu, cm0, j), pj1 = __shfl_sync(0xffffffffu, cm1, j);
            const unsigned pk0 = __shfl_sync(0xffffffffu, cm0, k), pk1 = __shfl_sync(0xffffffffu, cm1, k);
            bool oj0, oj1, ok0, ok1;
            decide(j, pj0, pj1, oj0, oj1);
            decide(k, two ? pk0 : 0u, two ? pk1 : 0u, ok0, ok1);
            push(j, oj0, oj1);
            if (two && !bad) push(k, ok0, ok1);
        }
        if (bD) fold();
        // A well-formed tree pushes each internal cell at most once per warp.
        if (bad || top == 0 || ++pops > max_pops) break;
        __syncwarp();
        if (K > 1 && shared && top >= kSplitAt) {   // each part keeps every K-th entry
            const int keep = (top - part + K - 1) / K;
            for (int i0 = 0; i0 < keep; i0 += 32) {
                const int i = i0 + lane;
                StackEntry e{0, 0, 0};
                if (i < keep) e = stk[w][i * K + part];
                __syncwarp();
                if (i < keep) stk[w][i] = e;
                __syncwarp();
            }
            top = keep;
            shared = false;
            mine = true;
            if (top == 0) break;
        }
        // ---- next step: up to 8 entries from the top of the stack ----
        // A step pushes at most 32 entries.  Above kMultiTop entries the walk
        // takes one entry per step, a depth-first walk that leaves at most 7
        // entries per tree level (7 * 21 + 8 in all), so the stack never holds
        // more than kMultiTop + 31 + 155 < kStack entries.
        const int cap = top <= kMultiTop ? 8 : 1;
        unsigned eF = 0, em0 = 0, em1 = 0;
        int en = 0;
        if (lane < cap && lane < top) {
            const StackEntry e = stk[w][top - 1 - lane];
            eF = (unsigned)e.range & ((1u << kRangeBits) - 1u);
            en = (int)((unsigned)e.range >> kRangeBits);
            em0 = (unsigned)e.lanes0;
            em1 = (unsigned)e.lanes1;
        }
        int incl = en;   // inclusive prefix of the child counts over lanes 0..7
        for (int o = 1; o < 8; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const unsigned take = __ballot_sync(0xffffffffu, lane < cap && lane < top && incl <= 32);
        const int P = __popc(take);   // >= 1: an entry has at most 8 children
        T = __shfl_sync(0xffffffffu, incl, P - 1);
        __syncwarp();
        top -= P;
        // this lane's entry: the last taken entry whose children start at or
        // before it (every entry has at least one child, so the starts differ)
        const unsigned starts = __reduce_or_sync(0xffffffffu, lane < P ? 1u << (incl - en) : 0u);
        const int q = (__popc(starts & ((2u << lane) - 1u)) - 1) & 7;
        const unsigned qF = __shfl_sync(0xffffffffu, eF, q);
        const int qx = __shfl_sync(0xffffffffu, incl - en, q);
        cm0 = __shfl_sync(0xffffffffu, em0, q);
        cm1 = __shfl_sync(0xffffffffu, em1, q);
        ch = qF + (unsigned)(lane - qx);
        if (K > 1) {
            fetch();
            if (nf + np > kList - 32) flush();   // a step adds at most 32
        }
    }
    if (!bad) flush();
    if ((bad || top > 0) && lane == 0) record_error(err, DEV_STACK_OVERFLOW);
    if (K > 1) {
        // the parts' sums, added in order by part 0
        float* mysum = reinterpret_cast<float*>(ls_src[w]);
        __syncwarp();
        if (part > 0) {
            const float v[12] = {sx.x, sy.x, sz.x, cx.x, cy.x, cz.x, sx.y, sy.y, sz.y, cx.y, cy.y, cz.y};   // c negated
#pragma unroll
            for (int k = 0; k < 12; ++k) mysum[k * 32 + lane] = v[k];
        }
        __syncthreads();
        if (part == 0) {
            // (either sum may be the larger, which a Kahan addition does not allow for)
            auto add = [&](float& s, float& c, float o, float oc) {
                float e;
                s = two_sum(s, o, e);
                c = (c + oc) + e;
            };
            for (int q = 1; q < K; ++q) {
                const float* o = reinterpret_cast<const float*>(ls_src[w + q]) + lane;
                add(sx.x, cx.x, o[0], o[96]); add(sy.x, cy.x, o[32], o[128]); add(sz.x, cz.x, o[64], o[160]);
                add(sx.y, cx.y, o[192], o[288]); add(sy.y, cy.y, o[224], o[320]); add(sz.y, cz.y, o[256], o[352]);
            }
        }
    }
    if (part == 0) {
        if (v0) acc[sorder[s0]] = make_float4(G * (sx.x + cx.x), G * (sy.x + cy.x), G * (sz.x + cz.x), 0.f);
        if (v1) acc[sorder[s1]] = make_float4(G * (sx.y + cx.y), G * (sy.y + cy.y), G * (sz.y + cz.y), 0.f);
    }
    unsigned long long c = cnt;
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if (lane == 0 && c) atomicAdd(inter, c);
}

}  // namespace nb
