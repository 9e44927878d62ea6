// nb_law.cuh -- the pairwise force law in FP32, shared by the direct-sum
// kernels (plain and batched).
//
// Reference law (Phys::Gravity, src/Sim/Physics.hpp:25-35, S = softening2):
//     a_i += m_j (p_j - p_i) / (r (r^2 + S)),   r = |p_j - p_i|
// with one MUFU.RSQ per pair: 1/(r (r^2+S)) = rsqrt(r^2 (r^2+S)^2 + tiny);
// tiny keeps the self pair's factor m rsqrt(tiny) finite, so that it adds
// exactly zero (times dp = 0).  tiny is 1e-30 unless the state's largest mass
// needs more (self_pair_tiny): masses above 1e21, as in the reference's own
// seeders (1e20..1e30), would make m * 1e15 overflow to inf and the self
// pair inf * 0 = NaN.  The raised tiny stays far below r^2 (r^2+S)^2 of any
// real pair at such scales.
// Plummer law: a_i += m_j (p_j - p_i) (r^2 + S)^{-3/2}.
#pragma once
#include "nb_common.cuh"
#include "../../include/nbody_gb300.h"

namespace nb {

constexpr int kFold = 32;            // sources summed in plain FP32 before a Kahan fold
constexpr float kTiny = 1e-30f;

// tiny for a state whose largest |mass| has the float bits *mmax_bits: the
// self pair's factor m / sqrt(tiny) stays <= 1e36 (1e-30 for masses <= 1e21).
__device__ __forceinline__ float self_pair_tiny(const unsigned* mmax_bits) {
    const float q = __uint_as_float(*mmax_bits) * 1e-36f;
    return fmaxf(kTiny, q * q);
}

template <int LAW>
__device__ __forceinline__ void interact(const float4 pj, float xi, float yi, float zi, float S, float tiny,
                                         float& ax, float& ay, float& az) {
    float dx = pj.x - xi;
    float dy = pj.y - yi;
    float dz = pj.z - zi;
    if (LAW == NB_LAW_REFERENCE) {
        float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
        float s = r2 + S;
        float t = fmaf(r2 * s, s, tiny);
        float w = pj.w * rsqrt_approx(t);
        ax = fmaf(w, dx, ax);
        ay = fmaf(w, dy, ay);
        az = fmaf(w, dz, az);
    } else {
        float q = fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, S)));
        float inv = rsqrt_approx(q);
        float w = pj.w * inv * (inv * inv);
        ax = fmaf(w, dx, ax);
        ay = fmaf(w, dy, ay);
        az = fmaf(w, dz, az);
    }
}

// The same interaction for two target bodies at once with the packed FP32x2
// instructions of sm_100+ (FADD2 / FMUL2 / FFMA2): identical operations in
// identical order, half the issue slots.  n* hold the negated target
// coordinates, so dx = xj + (-xi) rounds exactly like xj - xi.
template <int LAW>
__device__ __forceinline__ void interact_x2(float2 jx, float2 jy, float2 jz, float2 jm, float2 nx, float2 ny,
                                            float2 nz, float2 S2, float2 T2, float2& ax, float2& ay, float2& az) {
    const float2 dx = __fadd2_rn(jx, nx);
    const float2 dy = __fadd2_rn(jy, ny);
    const float2 dz = __fadd2_rn(jz, nz);
    float2 w;
    if (LAW == NB_LAW_REFERENCE) {
        float2 r2 = __fmul2_rn(dx, dx);
        r2 = __ffma2_rn(dy, dy, r2);
        r2 = __ffma2_rn(dz, dz, r2);
        const float2 s = __fadd2_rn(r2, S2);
        const float2 t = __ffma2_rn(__fmul2_rn(r2, s), s, T2);
        w = __fmul2_rn(jm, make_float2(rsqrt_approx(t.x), rsqrt_approx(t.y)));
    } else {
        float2 q = __ffma2_rn(dx, dx, S2);
        q = __ffma2_rn(dy, dy, q);
        q = __ffma2_rn(dz, dz, q);
        const float2 inv = make_float2(rsqrt_approx(q.x), rsqrt_approx(q.y));
        w = __fmul2_rn(__fmul2_rn(jm, inv), __fmul2_rn(inv, inv));
    }
    ax = __ffma2_rn(w, dx, ax);
    ay = __ffma2_rn(w, dy, ay);
    az = __ffma2_rn(w, dz, az);
}

// The factors of the separation for both bodies of two pairs at once: wi, with
// the mass jm of one body, is the acceleration of the other, and wj, with mi, its
// own.  Under the Plummer law a mass enters before the cube of the inverse
// distance is complete, as in interact_x2: the cube alone leaves FP32's range
// beyond 4e12 length units (and with a softening below 1e-13), far inside that
// of the factor (states in metres and kilograms, or in very small units).
template <int LAW>
__device__ __forceinline__ void pair_factors_x2(float2 dx, float2 dy, float2 dz, float2 S2, float2 T2, float2 jm,
                                                float2 mi, float2& wi, float2& wj) {
    if (LAW == NB_LAW_REFERENCE) {
        float2 r2 = __fmul2_rn(dx, dx);
        r2 = __ffma2_rn(dy, dy, r2);
        r2 = __ffma2_rn(dz, dz, r2);
        const float2 s = __fadd2_rn(r2, S2);
        const float2 t = __ffma2_rn(__fmul2_rn(r2, s), s, T2);
        const float2 w = make_float2(rsqrt_approx(t.x), rsqrt_approx(t.y));
        wi = __fmul2_rn(jm, w);
        wj = __fmul2_rn(mi, w);
        return;
    }
    float2 q = __ffma2_rn(dx, dx, S2);
    q = __ffma2_rn(dy, dy, q);
    q = __ffma2_rn(dz, dz, q);
    const float2 inv = make_float2(rsqrt_approx(q.x), rsqrt_approx(q.y));
    const float2 inv2 = __fmul2_rn(inv, inv);
    wi = __fmul2_rn(__fmul2_rn(jm, inv), inv2);
    wj = __fmul2_rn(__fmul2_rn(mi, inv), inv2);
}

// kahan_add of two sums at once in packed instructions (the same roundings);
// nc holds the negated compensations: the represented values are s + nc.
__device__ __forceinline__ void kahan_add_x2(float2& s, float2& nc, float2 x) {
    const float2 minus = make_float2(-1.f, -1.f);
    const float2 y = __fadd2_rn(x, nc);
    const float2 t = __fadd2_rn(s, y);
    nc = __ffma2_rn(__ffma2_rn(s, minus, t), minus, y);   // y - (t - s), each product exact
    s = t;
}

// Consecutive threads that fold one body's partials together.
constexpr int kFoldLanes = 8;

// Knuth's two-sum: s + b as a rounded sum and its exact error, whichever is larger.
__device__ __forceinline__ float two_sum(float s, float b, float& err) {
    const float t = __fadd_rn(s, b), u = __fsub_rn(t, s);
    err = __fadd_rn(__fsub_rn(s, __fsub_rn(t, u)), __fsub_rn(b, u));
    return t;
}

// Sum over the fold's lanes of (s - c), the same in every lane: added pairwise
// with the rounding error of each sum carried in the low part; the total is hi + lo, hi its rounding to a few units.
struct HiLo {
    float hi, lo;
    __device__ __forceinline__ float rounded() const { return __fadd_rn(hi, lo); }
};
struct HiLo3 {
    HiLo x, y, z;
    __device__ __forceinline__ float3 rounded() const { return make_float3(x.rounded(), y.rounded(), z.rounded()); }
};

__device__ __forceinline__ HiLo butterfly_total(float s, float c) {
    float hi = s, lo = -c;
#pragma unroll
    for (int o = 1; o < kFoldLanes; o <<= 1) {
        const float b = __shfl_xor_sync(0xffffffffu, hi, o);
        const float bl = __shfl_xor_sync(0xffffffffu, lo, o);
        float e;   // the sum's error is exact, so either side of the exchange finds the same
        hi = two_sum(hi, b, e);
        lo = __fadd_rn(__fadd_rn(lo, bl), e);
    }
    return HiLo{hi, lo};
}

// The warps of a block that fold the partials of 32 bodies together (body =
// lane: neighbouring entries are read together) each bring a compensated sum
// (s, c); the first warp's threads get the totals, added in the warps' order with
// the rounding errors carried.  Every thread of the block calls it.
constexpr int kFoldWarps = 8;
__device__ __forceinline__ HiLo3 add_warps(float (*sums)[6][32], float ax, float ay, float az, float kx, float ky,
                                            float kz) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    sums[w][0][lane] = ax; sums[w][1][lane] = ay; sums[w][2][lane] = az;
    sums[w][3][lane] = kx; sums[w][4][lane] = ky; sums[w][5][lane] = kz;
    __syncthreads();
    HiLo r[3] = {};
    if (w == 0) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            r[d] = HiLo{sums[0][d][lane], -sums[0][3 + d][lane]};
#pragma unroll
            for (int v = 1; v < kFoldWarps; ++v) {
                float e;
                r[d].hi = two_sum(r[d].hi, sums[v][d][lane], e);
                r[d].lo += e - sums[v][3 + d][lane];
            }
        }
    }
    return HiLo3{r[0], r[1], r[2]};
}

// One warp's evaluation of a chunk of 32 sources (in shared memory) against its
// 32 * IPT targets (IPT a lane in registers, negated coordinates nx, ny, nz and
// masses mi, packed in pairs).  BOTH: each pair serves both bodies, 17 FP32
// operations for two interactions instead of 26: lane l takes source
// (l + r) mod 32 at step r, and the sources' sums travel with them by shuffle;
// lane l receives source l's sum in out.  Else only the targets' side.  The
// chunk's target sums are added to the compensated sum (x, y, z of target k at
// 3 k, comp negated).
constexpr int kDirChunk = 32;
template <int LAW, int IPT, bool BOTH>
__device__ __forceinline__ void direct_chunk(const float4* src, int lane, const float2* nx, const float2* ny,
                                             const float2* nz, const float2* mi, float2 S2, float2 T2, float* sum,
                                             float* comp, float3& out) {
    constexpr int P = IPT / 2, kGroup = 4;
    const float2 z2 = make_float2(0.f, 0.f);
    float2 ax[P], ay[P], az[P];
#pragma unroll
    for (int q = 0; q < P; ++q) ax[q] = ay[q] = az[q] = z2;
    float sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll 1
    for (int g = 0; g < kDirChunk; g += kGroup) {
        float2 bx = z2, by = z2, bz = z2;
#pragma unroll
        for (int u = 0; u < kGroup; ++u) {
            const float4 pj = src[(lane + g + u) & 31];
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
                if (BOTH) {
                    bx = __ffma2_rn(wj, dx, bx);
                    by = __ffma2_rn(wj, dy, by);
                    bz = __ffma2_rn(wj, dz, bz);
                }
            }
            if (BOTH && u + 1 < kGroup) {
                const int next = (lane + 1) & 31;
                bx.x = __shfl_sync(0xffffffffu, bx.x, next); bx.y = __shfl_sync(0xffffffffu, bx.y, next);
                by.x = __shfl_sync(0xffffffffu, by.x, next); by.y = __shfl_sync(0xffffffffu, by.y, next);
                bz.x = __shfl_sync(0xffffffffu, bz.x, next); bz.y = __shfl_sync(0xffffffffu, bz.y, next);
            }
        }
        if (BOTH) {   // the source's earlier groups were left kGroup lanes on
            const int from = (lane + kGroup) & 31;
            sx = __shfl_sync(0xffffffffu, sx, from) + (bx.x + bx.y);
            sy = __shfl_sync(0xffffffffu, sy, from) + (by.x + by.y);
            sz = __shfl_sync(0xffffffffu, sz, from) + (bz.x + bz.y);
        }
    }
#pragma unroll
    for (int q = 0; q < P; ++q) {
        kahan_add(sum[6 * q], comp[6 * q], ax[q].x);
        kahan_add(sum[6 * q + 1], comp[6 * q + 1], ay[q].x);
        kahan_add(sum[6 * q + 2], comp[6 * q + 2], az[q].x);
        kahan_add(sum[6 * q + 3], comp[6 * q + 3], ax[q].y);
        kahan_add(sum[6 * q + 4], comp[6 * q + 4], ay[q].y);
        kahan_add(sum[6 * q + 5], comp[6 * q + 5], az[q].y);
    }
    if (BOTH) {   // lane l holds source (l + 31) mod 32
        const int own = (lane + 1) & 31;
        out = make_float3(-__shfl_sync(0xffffffffu, sx, own), -__shfl_sync(0xffffffffu, sy, own),
                          -__shfl_sync(0xffffffffu, sz, own));
    }
}

}  // namespace nb
