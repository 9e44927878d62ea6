// nb_fp64.cu -- FP64 direct-sum oracle (K8) and FP64 diagnostics.
//
// The FP64 oracle measures force error: for m sampled target bodies it
// sums the exact force law in double precision over all n sources, from the
// same float positions and masses the FP32 kernels use.  The diagnostics
// reduce kinetic energy, linear and angular momentum, mass and centre of mass
// in FP64; the O(n^2) potential evaluates each pair term in FP32, once, and
// accumulates it in FP64.  All reductions write per-block partials that one
// block folds in a fixed order, so results are deterministic.
#include "nb_common.cuh"
#include "nb_internal.hpp"
#include <algorithm>
#include <cmath>

namespace nb {

constexpr int kF64Block = 256;
constexpr int kF64Targets = 8;

template <int LAW>
__global__ void __launch_bounds__(kF64Block) k_fp64_forces(const float4* __restrict__ pos, int n,
                                                            const int32_t* __restrict__ targets, int m, double S,
                                                            double G, double* __restrict__ out3) {
    __shared__ double red[kF64Targets][3][kF64Block / 32];
    const int t0 = blockIdx.x * kF64Targets;
    double xi[kF64Targets], yi[kF64Targets], zi[kF64Targets];
    int ii[kF64Targets];
    double fx[kF64Targets], fy[kF64Targets], fz[kF64Targets];
#pragma unroll
    for (int k = 0; k < kF64Targets; ++k) {
        const int t = min(t0 + k, m - 1);
        ii[k] = targets[t];
        const float4 p = pos[ii[k]];
        xi[k] = p.x; yi[k] = p.y; zi[k] = p.z;
        fx[k] = fy[k] = fz[k] = 0.0;
    }
    for (int j = threadIdx.x; j < n; j += kF64Block) {
        const float4 pj = pos[j];
#pragma unroll
        for (int k = 0; k < kF64Targets; ++k) {
            const double dx = (double)pj.x - xi[k], dy = (double)pj.y - yi[k], dz = (double)pj.z - zi[k];
            const double r2 = dx * dx + dy * dy + dz * dz;
            double w;
            if (LAW == NB_LAW_REFERENCE) w = (double)pj.w / (sqrt(r2) * (r2 + S));
            else { const double q = r2 + S; w = (double)pj.w / (q * sqrt(q)); }
            if (j == ii[k] || r2 == 0.0) w = 0.0;
            fx[k] += w * dx; fy[k] += w * dy; fz[k] += w * dz;
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < kF64Targets; ++k) {
        double a = fx[k], b = fy[k], c = fz[k];
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_down_sync(0xffffffffu, a, o);
            b += __shfl_down_sync(0xffffffffu, b, o);
            c += __shfl_down_sync(0xffffffffu, c, o);
        }
        if (lane == 0) { red[k][0][warp] = a; red[k][1][warp] = b; red[k][2][warp] = c; }
    }
    __syncthreads();
    if (threadIdx.x < kF64Targets * 3) {
        const int k = threadIdx.x / 3, c = threadIdx.x % 3;
        if (t0 + k < m) {
            double s = 0.0;
            for (int w = 0; w < kF64Block / 32; ++w) s += red[k][c][w];
            const float mi = pos[ii[k]].w;
            out3[(size_t)(t0 + k) * 3 + c] = G * (double)mi * s;
        }
    }
}

// Per-body FP64 terms: K, p, L, M, m*x.
constexpr int kDiagTerms = 11;   // K px py pz Lx Ly Lz M mx my mz; U follows in the result

__global__ void __launch_bounds__(kF64Block) k_diag_partial(const float4* __restrict__ pos,
                                                             const float4* __restrict__ posc,
                                                             const float4* __restrict__ vel,
                                                             const float4* __restrict__ velc,
                                                             const float4* __restrict__ acc, float half_dt, int n,
                                                             double* __restrict__ partial) {
    __shared__ double red[kDiagTerms][kF64Block / 32];
    const int i = blockIdx.x * kF64Block + threadIdx.x;
    const float4 pi = pos[i];   // i < n_pad always (grid covers n_pad exactly)
    double term[kDiagTerms];
#pragma unroll
    for (int k = 0; k < kDiagTerms; ++k) term[k] = 0.0;
    if (i < n) {
        const float4 xc = posc[i], v = vel[i], vc = velc[i];
        const double m = pi.w;
        const double x = (double)pi.x - xc.x, y = (double)pi.y - xc.y, z = (double)pi.z - xc.z;
        double vx = (double)v.x - vc.x, vy = (double)v.y - vc.y, vz = (double)v.z - vc.z;
        if (acc) {
            const float4 a = acc[i];
            vx += (double)a.x * half_dt; vy += (double)a.y * half_dt; vz += (double)a.z * half_dt;
        }
        term[0] = 0.5 * m * (vx * vx + vy * vy + vz * vz);
        term[1] = m * vx; term[2] = m * vy; term[3] = m * vz;
        term[4] = m * (y * vz - z * vy);
        term[5] = m * (z * vx - x * vz);
        term[6] = m * (x * vy - y * vx);
        term[7] = m;
        term[8] = m * x; term[9] = m * y; term[10] = m * z;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < kDiagTerms; ++k) {
        double a = term[k];
        for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
        if (lane == 0) red[k][warp] = a;
    }
    __syncthreads();
    if (threadIdx.x < kDiagTerms) {
        double s = 0.0;
        for (int w = 0; w < kF64Block / 32; ++w) s += red[threadIdx.x][w];
        partial[(size_t)blockIdx.x * kDiagTerms + threadIdx.x] = s;
    }
}

// ---- pair potential ---------------------------------------------------------
// The pair function of two targets and one source: atan(eps / r) under the
// reference law (pi/2 - atan(r / eps)), (r^2 + S)^-1/2 under the Plummer law.
// (A packed FP32x2 series for distant pairs took 0.35 instead of 0.49 ms at
// 32,768 bodies, but 1.4 times the error of the sum.)
template <int LAW>
__device__ __forceinline__ float2 pair_potential(float2 r2, float2 eps2, float2 S2) {
    if (LAW == NB_LAW_REFERENCE) {
        const float2 x = __fmul2_rn(eps2, make_float2(rsqrtf(r2.x), rsqrtf(r2.y)));
        return make_float2(atanf(x.x), atanf(x.y));
    }
    const float2 q = __fadd2_rn(r2, S2);
    return make_float2(rsqrtf(q.x), rsqrtf(q.y));
}

// Blocks of kF64Block bodies, B of them (even): block b takes the pairs of its
// bodies with those of blocks b + d (mod B), d = 1 .. B/2 - 1, of block
// b + B/2 when b < B/2, and of itself at half weight (both orders): every
// unordered pair of bodies once, the same work in every block.  The offsets d
// are cut into gridDim.y runs, so that small states fill the GPU too.  Bound by
// instruction issue (the arc tangent).  GB300, with the rest of nb_diagnostics:
// 32,768 bodies 1.72 -> 0.55 ms (it evaluated both orders of every pair on 128
// blocks, and mapped memory for its result), 1,048,576 bodies 1.04 -> 0.48 s.
constexpr int kPotThreads = kF64Block / 2;   // two targets a thread
constexpr int kPotGroup = 64;                // terms summed in FP32 before FP64
template <int LAW>
__global__ void __launch_bounds__(kPotThreads) k_diag_potential(const float4* __restrict__ pos, int n, int nblocks, float eps,
                                                                float S, double* __restrict__ partial) {
    __shared__ float4 tile[kF64Block];
    __shared__ double red[kPotThreads / 32];
    const int tid = threadIdx.x, b = blockIdx.x;
    const float4 p0 = pos[b * kF64Block + tid], p1 = pos[b * kF64Block + kPotThreads + tid];
    const float2 nx = make_float2(-p0.x, -p1.x), ny = make_float2(-p0.y, -p1.y), nz = make_float2(-p0.z, -p1.z);
    const float2 eps2 = make_float2(eps, eps), S2 = make_float2(S, S);
    const int last = nblocks / 2 - (b < nblocks / 2 ? 0 : 1);   // largest offset of this block
    const int per = (nblocks / 2 + 1 + gridDim.y - 1) / gridDim.y;
    const int d0 = blockIdx.y * per, d1 = min(last + 1, d0 + per);
    double u0 = 0.0, u1 = 0.0;
    for (int d = d0; d < d1; ++d) {
        const int t = (b + d) % nblocks;
        __syncthreads();
        tile[tid] = pos[t * kF64Block + tid];
        tile[tid + kPotThreads] = pos[t * kF64Block + kPotThreads + tid];
        __syncthreads();
        double v0 = 0.0, v1 = 0.0;
        for (int g = 0; g < kF64Block; g += kPotGroup) {
            float2 s = make_float2(0.f, 0.f);
#pragma unroll 4
            for (int k = 0; k < kPotGroup; ++k) {
                const float4 pj = tile[g + k];
                const float2 dx = __fadd2_rn(make_float2(pj.x, pj.x), nx);
                const float2 dy = __fadd2_rn(make_float2(pj.y, pj.y), ny);
                const float2 dz = __fadd2_rn(make_float2(pj.z, pj.z), nz);
                const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                float2 phi = pair_potential<LAW>(r2, eps2, S2);
                if (d == 0) {   // the body itself (infinite where S underflows in FP32)
                    if (g + k == tid) phi.x = 0.f;
                    if (g + k == tid + kPotThreads) phi.y = 0.f;
                }
                s = __ffma2_rn(make_float2(pj.w, pj.w), phi, s);
            }
            v0 += (double)s.x;
            v1 += (double)s.y;
        }
        const double weight = d == 0 ? 0.5 : 1.0;
        u0 += weight * v0;
        u1 += weight * v1;
    }
    if (b * kF64Block + tid >= n) u0 = 0.0;   // padding
    if (b * kF64Block + kPotThreads + tid >= n) u1 = 0.0;
    double u = (double)p0.w * u0 + (double)p1.w * u1;
    for (int o = 16; o > 0; o >>= 1) u += __shfl_down_sync(0xffffffffu, u, o);
    if ((tid & 31) == 0) red[tid >> 5] = u;
    __syncthreads();
    if (tid == 0) {
        double sum = 0.0;
        for (int w = 0; w < kPotThreads / 32; ++w) sum += red[w];
        partial[(size_t)blockIdx.y * nblocks + b] = (LAW == NB_LAW_REFERENCE) ? -sum / (double)eps : -sum;
    }
}

// out: the folded terms, then G times the folded potential.
__global__ void k_diag_final(const double* __restrict__ partial, int nblocks, const double* __restrict__ potential,
                             int npot, double G, double* __restrict__ out) {
    __shared__ double red[kDiagTerms + 1][32];
    const int k = threadIdx.x / 32, lane = threadIdx.x % 32;
    double s = 0.0;
    if (k < kDiagTerms) {
        for (int b = lane; b < nblocks; b += 32) s += partial[(size_t)b * kDiagTerms + k];
    } else {
#pragma unroll 4
        for (int b = lane; b < npot; b += 32) s += potential[b];
    }
    red[k][lane] = s;
    __syncthreads();
    if (threadIdx.x <= kDiagTerms) {
        double t = 0.0;
        for (int l = 0; l < 32; ++l) t += red[threadIdx.x][l];
        out[threadIdx.x] = (threadIdx.x == kDiagTerms) ? G * t : t;
    }
}

cudaError_t fp64_forces(nb_sim* sim, const int32_t* d_targets, size_t m, double* d_out3) {
    if (m == 0) return cudaSuccess;
    const int blocks = (int)((m + kF64Targets - 1) / kF64Targets);
    if (sim->prm.law == NB_LAW_PLUMMER)
        k_fp64_forces<NB_LAW_PLUMMER><<<blocks, kF64Block, 0, sim->stream>>>(
            sim->pos, (int)sim->n, d_targets, (int)m, sim->prm.softening2, sim->prm.G, d_out3);
    else
        k_fp64_forces<NB_LAW_REFERENCE><<<blocks, kF64Block, 0, sim->stream>>>(
            sim->pos, (int)sim->n, d_targets, (int)m, sim->prm.softening2, sim->prm.G, d_out3);
    return cudaGetLastError();
}

// out: [K, px, py, pz, Lx, Ly, Lz, M, mx, my, mz, U]
cudaError_t fp64_diagnostics_ex(nb_sim* sim, float half_dt, bool with_acc, bool with_potential, double* d_out) {
    const int nblocks = (int)(sim->n_pad / kF64Block);
    static_assert(kPad / kF64Block % 2 == 0, "an even number of blocks");
    // runs of offsets: about 16 blocks of 128 threads an SM
    const int runs = std::max(1, std::min(nblocks / 2 + 1, (16 * std::max(1, sim->sm_count) + nblocks - 1) / nblocks));
    const size_t terms = (size_t)nblocks * kDiagTerms, need = terms + (size_t)nblocks * runs;
    if (need > sim->dscratch_cap) {
        dev_free(sim->dscratch, sim->stream);
        sim->dscratch = nullptr;
        sim->dscratch_cap = 0;
        cudaError_t e = dev_alloc(&sim->dscratch, need * sizeof(double));
        if (e != cudaSuccess) return e;
        sim->dscratch_cap = need;
    }
    const float eps = (float)sqrt(sim->prm.softening2);
    const float S = (float)sim->prm.softening2;
    double* potential = sim->dscratch + terms;
    k_diag_partial<<<nblocks, kF64Block, 0, sim->stream>>>(sim->pos, sim->posc, sim->vel, sim->velc,
                                                          with_acc ? sim->acc : nullptr, half_dt, (int)sim->n,
                                                          sim->dscratch);
    if (with_potential) {
        const dim3 grid((unsigned)nblocks, (unsigned)runs);
        if (sim->prm.law == NB_LAW_PLUMMER)
            k_diag_potential<NB_LAW_PLUMMER><<<grid, kPotThreads, 0, sim->stream>>>(sim->pos, (int)sim->n, nblocks, eps, S, potential);
        else
            k_diag_potential<NB_LAW_REFERENCE><<<grid, kPotThreads, 0, sim->stream>>>(sim->pos, (int)sim->n, nblocks, eps, S,
                                                                                      potential);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_diag_final<<<1, 32 * (kDiagTerms + 1), 0, sim->stream>>>(sim->dscratch, nblocks, potential,
                                                               with_potential ? nblocks * runs : 0, sim->prm.G, d_out);
    return cudaGetLastError();
}

cudaError_t fp64_diagnostics(nb_sim* sim, double* d_out) { return fp64_diagnostics_ex(sim, 0.f, false, true, d_out); }

}  // namespace nb
