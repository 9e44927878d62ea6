// nb_api.cu -- the C-ABI of the N-body step (include/nbody_gb300.h).
//
// Host side of the drop-in boundary for INBodySim (src/Sim/INBodySim.hpp:19-25):
// handle management, uploads of the reference's 104-byte Particle records
// (unpacked on the GPU), the step loop, and the write-back of Position,
// Velocity and Forces.  Every call returns a status code; messages are kept
// per handle (nb_last_error).
#include "nb_common.cuh"
#include "nb_internal.hpp"
#include "nb_refseed.hpp"
#include <cmath>
#include <cstring>
#include <cstdio>
#include <new>
#include <string>
#include <thread>
#include <vector>
#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>

using namespace nb;

namespace {

static_assert(sizeof(nb_particle) == 104, "nb_particle must match the reference's 104-byte record");
static_assert(offsetof(nb_particle, velocity) == 48, "Velocity at offset 48");
static_assert(offsetof(nb_particle, forces) == 72, "Forces at offset 72");
static_assert(offsetof(nb_particle, mass) == 96, "Mass at offset 96");
static_assert(sizeof(nb_render_vertex) == 32, "LWParticle is 32 bytes");

// Packed write-back record: position, velocity, force.
struct WbRecord {
    float pos[3];
    float pad;
    double vel[3];
    double force[3];
};
static_assert(sizeof(WbRecord) == 64, "write-back record is 64 bytes");

int fail(nb_sim* s, int code, const std::string& msg) {
    if (s) s->err = msg;
    return code;
}

int cuda_fail(nb_sim* s, cudaError_t e, const char* where) {
    if (s) s->err = std::string(where) + ": " + cudaGetErrorString(e);
    return NB_ECUDA;
}

#define NB_CUDA(sim, call)                                           \
    do {                                                             \
        cudaError_t e_ = (call);                                     \
        if (e_ != cudaSuccess) return cuda_fail((sim), e_, #call);   \
    } while (0)

// Unpacks reference records into the SoA state; flags non-finite input.
__global__ void k_unpack_records(const nb_particle* __restrict__ in, int n, int kind, float4* __restrict__ pos,
                                 float4* __restrict__ posc, float4* __restrict__ vel, float4* __restrict__ velc,
                                 float4* __restrict__ finit, int* __restrict__ any_force, int* __restrict__ err,
                                 unsigned* __restrict__ mmax) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const nb_particle& p = in[i];
    const float m = (float)p.mass;
    if (isfinite(m)) atomicMax(mmax, __float_as_uint(fabsf(m)));
    const float ext = fmaxf(fmaxf(fabsf(p.position[0]), fabsf(p.position[1])), fabsf(p.position[2]));
    if (isfinite(ext)) atomicMax(mmax + 1, __float_as_uint(ext));
    pos[i] = make_float4(p.position[0], p.position[1], p.position[2], m);
    posc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    vel[i] = make_float4((float)p.velocity[0], (float)p.velocity[1], (float)p.velocity[2], 0.f);
    // Low part of the double velocity kept as the Kahan compensation (value = v - c).
    velc[i] = make_float4((float)((double)(float)p.velocity[0] - p.velocity[0]),
                          (float)((double)(float)p.velocity[1] - p.velocity[1]),
                          (float)((double)(float)p.velocity[2] - p.velocity[2]), 0.f);
    bool finite = isfinite(p.position[0]) && isfinite(p.position[1]) && isfinite(p.position[2]) &&
                  isfinite(p.velocity[0]) && isfinite(p.velocity[1]) && isfinite(p.velocity[2]) &&
                  isfinite(p.mass) && isfinite(p.forces[0]) && isfinite(p.forces[1]) && isfinite(p.forces[2]);
    if (!finite) record_error(err, DEV_BAD_INPUT);
    // BruteForceCPU adds onto the records' Forces (src/Sim/BruteForceCPU.cpp:40);
    // keep any initial force as an acceleration applied by the first step.
    if (kind != NB_SIM_BARNES_HUT && finit) {
        const bool nz = p.forces[0] != 0.0 || p.forces[1] != 0.0 || p.forces[2] != 0.0;
        finit[i] = nz && p.mass != 0.0 ? make_float4((float)(p.forces[0] / p.mass), (float)(p.forces[1] / p.mass),
                                                     (float)(p.forces[2] / p.mass), 0.f)
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
        if (nz) atomicExch(any_force, 1);
    }
}

// Validates a state written by a copy (finite values), clears its
// compensation and records its largest |mass| in mmax[0] and its largest
// |coordinate| in mmax[1] (the caller cleared both).
__global__ void k_check_soa(const float4* __restrict__ pos, const float4* __restrict__ vel, int n,
                            float4* __restrict__ posc, float4* __restrict__ velc, int* __restrict__ err,
                            unsigned* __restrict__ mmax) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pos[i], v = vel[i];
    if (!(isfinite(p.x) && isfinite(p.y) && isfinite(p.z) && isfinite(p.w) && isfinite(v.x) && isfinite(v.y) &&
          isfinite(v.z)))
        record_error(err, DEV_BAD_INPUT);
    else {
        atomicMax(mmax, __float_as_uint(fabsf(p.w)));
        atomicMax(mmax + 1, __float_as_uint(fmaxf(fmaxf(fabsf(p.x), fabsf(p.y)), fabsf(p.z))));
    }
    posc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    velc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

__global__ void k_pack_writeback(const float4* __restrict__ pos, const float4* __restrict__ posc,
                                 const float4* __restrict__ vel, const float4* __restrict__ velc,
                                 const float4* __restrict__ acc, int n, int zero_forces,
                                 WbRecord* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pos[i], v = vel[i], vc = velc[i], a = acc[i];
    WbRecord r;
    r.pos[0] = p.x; r.pos[1] = p.y; r.pos[2] = p.z; r.pad = 0.f;
    r.vel[0] = (double)v.x - (double)vc.x;
    r.vel[1] = (double)v.y - (double)vc.y;
    r.vel[2] = (double)v.z - (double)vc.z;
    const double m = p.w;
    r.force[0] = zero_forces ? 0.0 : m * (double)a.x;
    r.force[1] = zero_forces ? 0.0 : m * (double)a.y;
    r.force[2] = zero_forces ? 0.0 : m * (double)a.z;
    out[i] = r;
}

// nb_write_back straight into the caller's records (host memory the GPU can
// address).  A warp rewrites its 32 records as one contiguous run, so that
// every store is coalesced into whole cache lines over the chip-to-chip link:
// Position, Velocity and Forces get the new values, all other words (colours,
// padding, mass) are read back and stored unchanged.  Bound by the link: its
// latency for few records, its rate for many.  So a warp has its whole run of
// loads in flight before its first store (16 bytes a load where the records
// are aligned to that), the fields are set in shared memory between, and the
// error word goes to the host beside the records, with no copy of its own.
// Word by word, each load behind the store before it, and a copy: 52 us for
// 1000 records, 51 for 4000, 103 for 100003, 897 for 2^20 (pageable records);
// this: 15, 17, 88 and 721 us.  Two blocks an SM keep the link's reads busy and
// spread the runs in time, so that reads and stores overlap: with all runs in
// flight at once 100003 records took 111 us and 262144 took 236, with two 197.
// A programmatic dependent launch behind the update (a 1000-body frame 22.4 us,
// now 20.0); nothing of the records is read before the wait: an earlier kernel
// of the stream may have written them.
constexpr int kRecWords = (int)(sizeof(nb_particle) / 4);   // 26
static_assert(sizeof(nb_particle) == 104, "reference record layout");
constexpr int kWbWarps = 2;                       // warps a block
constexpr int kWbPerSm = 2;                       // blocks an SM
constexpr int kWbVecs = 32 * kRecWords / 4;       // 16-byte words of a full run

__global__ void __launch_bounds__(32 * kWbWarps) k_writeback_records(
    const float4* pos, const float4* vel, const float4* velc, const float4* acc, int n, int zero_forces,
    uint32_t* out_words, const int* d_err, int* h_err) {
    wait_for_previous();
    __shared__ uint4 run4[kWbWarps][kWbVecs];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0) *h_err = *d_err;
    uint32_t* run = reinterpret_cast<uint32_t*>(run4[warp]);
    const bool aligned = (reinterpret_cast<uintptr_t>(out_words) & 15) == 0;   // a run is 3328 bytes
    const long long step = (long long)gridDim.x * kWbWarps * 32;
    for (long long base = ((long long)blockIdx.x * kWbWarps + warp) * 32; base < n; base += step) {
        const int nrec = (int)min(32LL, (long long)n - base), nwords = nrec * kRecWords;
        uint32_t* w0 = out_words + base * kRecWords;
        const bool wide = nrec == 32 && aligned;   // else word by word
        float4 p, v, vc, a;
        if (wide) {
            constexpr int PER = (kWbVecs + 31) / 32;
            const uint4* in = reinterpret_cast<const uint4*>(w0);
            uint4 q[PER];
#pragma unroll
            for (int k = 0; k < PER; ++k)
                if (lane + 32 * k < kWbVecs) q[k] = in[lane + 32 * k];
            p = pos[base + lane]; v = vel[base + lane]; vc = velc[base + lane]; a = acc[base + lane];
#pragma unroll
            for (int k = 0; k < PER; ++k)
                if (lane + 32 * k < kWbVecs) run4[warp][lane + 32 * k] = q[k];
        } else {
            uint32_t q[kRecWords];
#pragma unroll
            for (int k = 0; k < kRecWords; ++k)
                if (lane + 32 * k < nwords) q[k] = w0[lane + 32 * k];
            if (lane < nrec) { p = pos[base + lane]; v = vel[base + lane]; vc = velc[base + lane]; a = acc[base + lane]; }
#pragma unroll
            for (int k = 0; k < kRecWords; ++k)
                if (lane + 32 * k < nwords) run[lane + 32 * k] = q[k];
        }
        __syncwarp();
        if (lane < nrec) {
            float* f = reinterpret_cast<float*>(run + lane * kRecWords);
            f[0] = p.x; f[1] = p.y; f[2] = p.z;
            double* d = reinterpret_cast<double*>(f + 12);   // byte 48 of a 104-byte record: aligned
            const double m = p.w;
            d[0] = (double)v.x - (double)vc.x;
            d[1] = (double)v.y - (double)vc.y;
            d[2] = (double)v.z - (double)vc.z;
            d[3] = zero_forces ? 0.0 : m * (double)a.x;
            d[4] = zero_forces ? 0.0 : m * (double)a.y;
            d[5] = zero_forces ? 0.0 : m * (double)a.z;
        }
        __syncwarp();
        if (wide) {
            uint4* out = reinterpret_cast<uint4*>(w0);
            for (int j = lane; j < kWbVecs; j += 32) out[j] = run4[warp][j];
        } else {
            for (int j = lane; j < nwords; j += 32) w0[j] = run[j];
        }
        __syncwarp();
    }
}

__global__ void k_render_fill(const float4* __restrict__ pos, const float4* __restrict__ colour, float scale, int n,
                              nb_render_vertex* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pos[i];
    const float4 c = colour ? colour[i] : make_float4(1.f, 1.f, 1.f, 1.f);
    nb_render_vertex v;
    v.position[0] = p.x; v.position[1] = p.y; v.position[2] = p.z;
    v.colour[0] = c.x; v.colour[1] = c.y; v.colour[2] = c.z; v.colour[3] = c.w;
    v.scale = scale;
    out[i] = v;
}

// Kernels read and write the caller's records in place: the device reports
// that it addresses pageable host memory (Grace-attached GPUs do, over the
// coherent chip-to-chip link) and the caller did not ask for staged copies.
bool host_direct(const nb_sim* s) { return s->pageable_access == 1 && !(s->prm.flags & NB_FLAG_STAGED_IO); }

// Device / pinned host staging of at least `bytes`, reused across calls.
void* device_stage(nb_sim* s, size_t bytes) {
    if (bytes > s->d_stage_bytes) {
        cudaStreamSynchronize(s->stream);
        dev_free(s->d_stage, s->stream);
        s->d_stage = nullptr;
        s->d_stage_bytes = 0;
        if (dev_alloc(&s->d_stage, bytes) != cudaSuccess) {
            cudaGetLastError();
            s->d_stage = nullptr;
            return nullptr;
        }
        s->d_stage_bytes = bytes;
    }
    return s->d_stage;
}

void* host_stage(nb_sim* s, size_t bytes) {
    if (bytes > s->h_stage_bytes) {
        cudaStreamSynchronize(s->stream);
        if (s->h_stage) cudaFreeHost(s->h_stage);
        s->h_stage = nullptr;
        s->h_stage_bytes = 0;
        if (cudaMallocHost(&s->h_stage, bytes) != cudaSuccess) {
            cudaGetLastError();
            s->h_stage = nullptr;
            return nullptr;
        }
        s->h_stage_bytes = bytes;
    }
    return s->h_stage;
}

void detach_render(nb_sim* s) {
    cudaFree(s->render);
    cudaFree(s->rcolour);
    s->render = nullptr;
    s->rcolour = nullptr;
}

void free_state(nb_sim* s) {
    detach_render(s);
    for (void* p : {(void*)s->pos, (void*)s->posc, (void*)s->vel, (void*)s->velc, (void*)s->acc, (void*)s->finit,
                    (void*)s->part})
        dev_free(p, s->stream);
    s->pos = s->posc = s->vel = s->velc = s->acc = s->finit = s->part = nullptr;
    s->part_cap = 0;
    s->pair_cap = 0;
    s->cap = 0;
    tree_free(s);
}

int ensure_state(nb_sim* s, size_t n) {
    detach_render(s);   // a new particle set invalidates the vertex buffer (re-attach after Init)
    const size_t n_pad = pad_up(std::max<size_t>(n, 1), kPad);
    if (n_pad > s->cap) {
        free_state(s);
        const size_t bytes = n_pad * sizeof(float4);
        float4** arrs[] = {&s->pos, &s->posc, &s->vel, &s->velc, &s->acc, &s->finit};
        for (float4** a : arrs) {
            cudaError_t e = dev_alloc(a, bytes);
            if (e != cudaSuccess) {
                free_state(s);
                cudaGetLastError();
                return fail(s, NB_ENOMEM, std::string("device allocation failed: ") + cudaGetErrorString(e));
            }
        }
        s->cap = n_pad;
    }
    s->n = n;
    s->n_pad = n_pad;
    // zero the whole padded arrays: padded bodies are zero-mass at the origin
    const size_t bytes = s->cap * sizeof(float4);
    float4* arrs2[] = {s->pos, s->posc, s->vel, s->velc, s->acc, s->finit};
    for (float4* a : arrs2) NB_CUDA(s, cudaMemsetAsync(a, 0, bytes, s->stream));
    s->tree_valid = false;
    s->forces_fresh = false;
    s->finit_pending = false;
    return NB_OK;
}

// The device error word as copied to h_err[0] by a copy queued before the
// caller's last synchronisation of the stream.
int decode_device_error(nb_sim* s) {
    const int code = s->h_err[0];
    if (code == DEV_OK) return NB_OK;
    NB_CUDA(s, cudaMemsetAsync(s->d_err, 0, sizeof(int), s->stream));
    switch (code) {
        case DEV_WAIT_TIMEOUT: return fail(s, NB_ETIMEOUT, "a bounded device wait ran out; the step was abandoned");
        case DEV_STACK_OVERFLOW: return fail(s, NB_ENOTSUP, "tree traversal stack overflow (tree deeper than supported)");
        case DEV_TREE_OVERFLOW: return fail(s, NB_ENOMEM, "octree node capacity exceeded");
        case DEV_BAD_INPUT: return fail(s, NB_EINVAL, "non-finite value in the particle state");
        default: return fail(s, NB_ECUDA, "device error code " + std::to_string(code));
    }
}

// Whether the state's largest mass (h_err[2], read with the error word) needs
// the direct sum's heavy self-pair guard.
void note_masses(nb_sim* s) {
    float m;
    std::memcpy(&m, &s->h_err[2], sizeof(float));
    s->heavy = m > 1e21f;
}

int check_device_error(nb_sim* s) {
    NB_CUDA(s, cudaMemcpyAsync(s->h_err, s->d_err, sizeof(int), cudaMemcpyDeviceToHost, s->stream));
    NB_CUDA(s, cudaMemcpyAsync(s->h_err + 2, s->d_mmax, 2 * sizeof(unsigned), cudaMemcpyDeviceToHost, s->stream));
    NB_CUDA(s, cudaStreamSynchronize(s->stream));
    note_masses(s);
    return decode_device_error(s);
}

int force_pass(nb_sim* s, float dt, bool update) {
    if (s->prm.kind == NB_SIM_BARNES_HUT) {
        cudaError_t e = tree_build(s);
        if (e != cudaSuccess) return cuda_fail(s, e, "tree_build");
        e = tree_forces(s);
        if (e != cudaSuccess) return cuda_fail(s, e, "tree_forces");
        if (update) {
            e = kick_drift(s, dt);
            if (e != cudaSuccess) return cuda_fail(s, e, "kick_drift");
        }
    } else {
        cudaError_t e = direct_force_update(s, dt, update);
        if (e != cudaSuccess) return cuda_fail(s, e, "direct_force_update");
    }
    s->forces_fresh = !update;
    if (update) s->tree_valid = false;
    return NB_OK;
}

bool params_valid(const nb_params* p, std::string& why) {
    if (p->kind < 0 || p->kind > NB_SIM_BARNES_HUT) { why = "unknown simulator kind"; return false; }
    if (p->law != NB_LAW_REFERENCE && p->law != NB_LAW_PLUMMER) { why = "unknown force law"; return false; }
    if (!std::isfinite(p->G) || !std::isfinite(p->softening2) || p->softening2 < 0) { why = "bad G or softening2"; return false; }
    if (p->law == NB_LAW_PLUMMER && p->softening2 <= 0) { why = "Plummer law needs softening2 > 0"; return false; }
    if (!std::isfinite(p->theta) || p->theta < 0) { why = "bad theta"; return false; }
    if (!std::isfinite(p->pos_scale) || p->pos_scale == 0) { why = "bad pos_scale"; return false; }
    if (!(p->bounds_half > 0) || !std::isfinite(p->bounds_half)) { why = "bad bounds_half"; return false; }
    if (p->max_depth < 1 || p->max_depth > 21) { why = "max_depth must be 1..21"; return false; }
    if (p->leaf_size < 1 || p->leaf_size > 64) { why = "leaf_size must be 1..64"; return false; }
    return true;
}

}  // namespace

namespace nb {

struct DevicePool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;   // allocations are ordered on it, then waited for
};
static std::mutex g_pool_mu;
static std::map<int, DevicePool> g_pools;

cudaError_t dev_alloc(void** p, size_t bytes) {
    *p = nullptr;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(g_pool_mu);
    DevicePool& P = g_pools[dev];
    if (!P.pool) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        e = cudaMemPoolCreate(&P.pool, &props);
        if (e != cudaSuccess) { P.pool = nullptr; return e; }
        // keep freed memory in the pool for the next allocation
        uint64_t keep = UINT64_MAX;
        e = cudaMemPoolSetAttribute(P.pool, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&P.stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) {
            cudaMemPoolDestroy(P.pool);
            P.pool = nullptr;
            P.stream = nullptr;
            return e;
        }
    }
    e = cudaMallocFromPoolAsync(p, std::max<size_t>(bytes, 1), P.pool, P.stream);
    if (e != cudaSuccess) { *p = nullptr; return e; }
    // the allocation has taken place in stream order: usable on every stream
    e = cudaStreamSynchronize(P.stream);
    if (e != cudaSuccess) { cudaFreeAsync(*p, P.stream); *p = nullptr; }
    return e;
}

void dev_free(void* p, cudaStream_t st) {
    if (p) cudaFreeAsync(p, st);
}


int sim_reserve_zeroed(nb_sim* s, size_t n) {
    if (n > (size_t)INT32_MAX - kPad) return fail(s, NB_EINVAL, "too many particles");
    cudaSetDevice(s->dev);
    return ensure_state(s, n);
}

int sim_rescan_state(nb_sim* s) {
    cudaSetDevice(s->dev);
    if (s->n == 0) return NB_OK;
    NB_CUDA(s, cudaMemsetAsync(s->d_mmax, 0, 2 * sizeof(unsigned), s->stream));
    k_check_soa<<<(unsigned)((s->n + 255) / 256), 256, 0, s->stream>>>(s->pos, s->vel, (int)s->n, s->posc, s->velc,
                                                                      s->d_err, s->d_mmax);
    NB_CUDA(s, cudaGetLastError());
    return NB_OK;
}

int sim_check_state(nb_sim* s) {
    cudaSetDevice(s->dev);
    if (s->n == 0) return NB_OK;
    NB_CUDA(s, cudaMemsetAsync(s->d_mmax, 0, 2 * sizeof(unsigned), s->stream));
    k_check_soa<<<(unsigned)((s->n + 255) / 256), 256, 0, s->stream>>>(s->pos, s->vel, (int)s->n, s->posc, s->velc,
                                                                      s->d_err, s->d_mmax);
    NB_CUDA(s, cudaGetLastError());
    const int rc = check_device_error(s);
    if (rc) s->n = 0;
    return rc;
}

}  // namespace nb

extern "C" {

int nb_default_params(nb_params* p) {
    try {
        if (!p) return NB_EINVAL;
        std::memset(p, 0, sizeof(*p));
        p->kind = NB_SIM_BARNES_HUT;
        p->law = NB_LAW_REFERENCE;
        p->G = 1.0;
        p->softening2 = 1e-4;
        p->theta = 0.5;
        p->pos_scale = 1.0;
        p->bounds_half = 4000.0f;
        p->max_depth = 21;
        p->leaf_size = 1;
        p->device = 0;
        p->stream = nullptr;
        p->flags = NB_FLAG_NONE;
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

const char* nb_sim_name(int kind) {
    switch (kind) {
        case NB_SIM_BRUTE_FORCE: return "Brute Force CPU";
        case NB_SIM_BRUTE_FORCE_GPU: return "Brute Force GPU";
        case NB_SIM_BARNES_HUT: return "Barnes-Hut";
        default: return "Unknown";
    }
}

int nb_create(const nb_params* params, nb_sim** out) {
    try {
        if (!params || !out) return NB_EINVAL;
        *out = nullptr;
        std::string why;
        if (!params_valid(params, why)) return NB_EINVAL;
        nb_sim* s = new (std::nothrow) nb_sim();
        if (!s) return NB_ENOMEM;
        s->prm = *params;
        s->dev = params->device;
        int count = 0;
        if (cudaGetDeviceCount(&count) != cudaSuccess || count <= params->device || params->device < 0) {
            cudaGetLastError();
            delete s;
            return NB_ECUDA;
        }
        if (cudaSetDevice(s->dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&s->sm_count, cudaDevAttrMultiProcessorCount, s->dev) != cudaSuccess) {
            cudaGetLastError();
            delete s;
            return NB_ECUDA;
        }
        if (cudaDeviceGetAttribute(&s->pageable_access, cudaDevAttrPageableMemoryAccess, s->dev) != cudaSuccess) {
            cudaGetLastError();
            s->pageable_access = 0;
        }
        if (params->stream) {
            s->stream = (cudaStream_t)params->stream;
        } else {
            if (cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess) { delete s; return NB_ECUDA; }
            s->own_stream = true;
        }
        if (dev_alloc(&s->d_err, sizeof(int)) != cudaSuccess || cudaMallocHost(&s->h_err, 4 * sizeof(int)) != cudaSuccess ||
            dev_alloc(&s->d_inter, sizeof(unsigned long long)) != cudaSuccess ||
            dev_alloc(&s->d_mmax, 2 * sizeof(unsigned)) != cudaSuccess) {
            cudaGetLastError();
            nb_destroy(s);
            return NB_ENOMEM;
        }
        cudaMemsetAsync(s->d_err, 0, sizeof(int), s->stream);
        cudaMemsetAsync(s->d_inter, 0, sizeof(unsigned long long), s->stream);
        cudaMemsetAsync(s->d_mmax, 0, 2 * sizeof(unsigned), s->stream);
        s->h_err[0] = s->h_err[1] = s->h_err[2] = s->h_err[3] = 0;
        *out = s;
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_destroy(nb_sim* s) {
    try {
        if (!s) return NB_EINVAL;
        cudaSetDevice(s->dev);
        if (s->stream) cudaStreamSynchronize(s->stream);
        free_state(s);
        dev_free(s->d_stage, s->stream);
        if (s->h_stage) cudaFreeHost(s->h_stage);
        for (auto& p : s->prof.pending) { cudaEventDestroy(p.a); cudaEventDestroy(p.b); }
        for (cudaEvent_t e : s->prof.pool) cudaEventDestroy(e);
        dev_free(s->dscratch, s->stream);
        dev_free(s->d_err, s->stream);
        dev_free(s->d_inter, s->stream);
        dev_free(s->d_mmax, s->stream);
        if (s->h_err) cudaFreeHost(s->h_err);
        if (s->own_stream && s->stream) cudaStreamDestroy(s->stream);
        delete s;
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

const char* nb_last_error(const nb_sim* s) { return s ? s->err.c_str() : "null handle"; }

size_t nb_count(const nb_sim* s) { return s ? s->n : 0; }

void* nb_stream(nb_sim* s) { return s ? (void*)s->stream : nullptr; }

}  // extern "C"

namespace {

// Fills the records on the device: from the caller's host records (seeder < 0)
// or from one of the reference's seeders run on the GPU.
__global__ void k_seed_records(int seeder, uint64_t seed, float scale, nb::refseed::GalaxyFrame frame, int n,
                               nb_particle* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    nb_particle p;
    if (seeder == 0) nb::refseed::random_body(seed, (size_t)i, scale, p);
    else if (seeder == 1) nb::refseed::galaxy_body(seed, (size_t)i, scale, frame, p);
    else nb::refseed::star_system_body(seed, (size_t)i, p);
    out[i] = p;
}

// nb_init_particles / nb_init_seeded: records in host memory (host != null)
// or generated on the device, unpacked into the simulator's state.
int init_records(nb_sim* s, const nb_particle* host, int seeder, uint64_t seed, float scale, size_t n,
                 nb_particle* records_out) {
    if (n > (size_t)INT32_MAX - kPad) return fail(s, NB_EINVAL, "too many particles");
    cudaSetDevice(s->dev);
    int rc = ensure_state(s, n);
    if (rc) return rc;
    if (n == 0) return NB_OK;
    nb_particle* d_rec = static_cast<nb_particle*>(device_stage(s, n * sizeof(nb_particle) + 16));
    if (!d_rec) return fail(s, NB_ENOMEM, "device staging allocation failed");
    int* d_any = (int*)((char*)d_rec + n * sizeof(nb_particle));
    cudaError_t e = cudaSuccess;
    const nb_particle* src = d_rec;
    if (host) {   // the copy engine moves the records faster than kernel reads of host memory
        e = cudaMemcpyAsync(d_rec, host, n * sizeof(nb_particle), cudaMemcpyHostToDevice, s->stream);
    } else {
        const nb::refseed::GalaxyFrame frame = nb::refseed::galaxy_frame(seed, n);
        k_seed_records<<<(unsigned)((n + 255) / 256), 256, 0, s->stream>>>(seeder, seed, scale, frame, (int)n, d_rec);
        e = cudaGetLastError();
        if (e == cudaSuccess && records_out)
            e = cudaMemcpyAsync(records_out, d_rec, n * sizeof(nb_particle), cudaMemcpyDeviceToHost, s->stream);
    }
    if (e == cudaSuccess) e = cudaMemsetAsync(d_any, 0, sizeof(int), s->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(s->d_mmax, 0, 2 * sizeof(unsigned), s->stream);
    if (e == cudaSuccess) {
        k_unpack_records<<<(unsigned)((n + 255) / 256), 256, 0, s->stream>>>(src, (int)n, s->prm.kind, s->pos,
                                                                            s->posc, s->vel, s->velc, s->finit,
                                                                            d_any, s->d_err, s->d_mmax);
        e = cudaGetLastError();
    }
    // the force flag and the error word come back with one synchronisation
    int any = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(s->h_err + 1, d_any, sizeof(int), cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(s->h_err, s->d_err, sizeof(int), cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(s->h_err + 2, s->d_mmax, 2 * sizeof(unsigned), cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
    if (e == cudaSuccess) {
        any = s->h_err[1];
        note_masses(s);
    }
    if (e != cudaSuccess) return cuda_fail(s, e, host ? "nb_init_particles" : "nb_init_seeded");
    s->finit_pending = any != 0;
    rc = decode_device_error(s);
    if (rc) { s->n = 0; return rc; }
    return NB_OK;
}

}  // namespace

extern "C" {

int nb_init_particles(nb_sim* s, const nb_particle* particles, size_t n) {
    try {
        if (!s) return NB_EINVAL;
        if (!particles && n) return fail(s, NB_EINVAL, "null particle buffer");
        return init_records(s, particles, -1, 0, 1.f, n, nullptr);
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_init_seeded(nb_sim* s, int seeder, uint64_t seed, float scale, size_t n, nb_particle* records_out) {
    try {
        if (!s) return NB_EINVAL;
        if (seeder < 0 || seeder > 2 || !(scale > 0)) return fail(s, NB_EINVAL, "bad seeder or scale");
        return init_records(s, nullptr, seeder, seed, scale, n, records_out);
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_init_soa(nb_sim* s, const float* pos_mass4, const float* vel4, size_t n) {
    try {
        if (!s) return NB_EINVAL;
        if ((!pos_mass4 || !vel4) && n) return fail(s, NB_EINVAL, "null buffer");
        if (n > (size_t)INT32_MAX - kPad) return fail(s, NB_EINVAL, "too many particles");
        cudaSetDevice(s->dev);
        int rc = ensure_state(s, n);
        if (rc) return rc;
        if (n == 0) return NB_OK;
        NB_CUDA(s, cudaMemcpyAsync(s->pos, pos_mass4, n * sizeof(float4), cudaMemcpyHostToDevice, s->stream));
        NB_CUDA(s, cudaMemcpyAsync(s->vel, vel4, n * sizeof(float4), cudaMemcpyHostToDevice, s->stream));
        NB_CUDA(s, cudaMemsetAsync(s->d_mmax, 0, 2 * sizeof(unsigned), s->stream));
        k_check_soa<<<(unsigned)((n + 255) / 256), 256, 0, s->stream>>>(s->pos, s->vel, (int)n, s->posc, s->velc, s->d_err,
                                                                        s->d_mmax);
        NB_CUDA(s, cudaGetLastError());
        rc = check_device_error(s);
        if (rc) { s->n = 0; return rc; }
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_step(nb_sim* s, float dt, int nsteps) {
    try {
        if (!s) return NB_EINVAL;
        if (nsteps < 0 || !std::isfinite(dt)) return fail(s, NB_EINVAL, "bad dt or nsteps");
        if (s->n == 0) return NB_OK;
        cudaSetDevice(s->dev);
        for (int k = 0; k < nsteps; ++k) {
            int rc = force_pass(s, dt, true);
            if (rc) return rc;
        }
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_synchronize(nb_sim* s) {
    try {
        if (!s) return NB_EINVAL;
        cudaSetDevice(s->dev);
        return check_device_error(s);
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_read_state(nb_sim* s, float* pos3, double* vel3, double* force3) {
    try {
        if (!s) return NB_EINVAL;
        cudaSetDevice(s->dev);
        const size_t n = s->n;
        if (n == 0) return NB_OK;
        WbRecord* d_wb = static_cast<WbRecord*>(device_stage(s, n * sizeof(WbRecord)));
        WbRecord* h = static_cast<WbRecord*>(host_stage(s, n * sizeof(WbRecord)));
        if (!d_wb || !h) return fail(s, NB_ENOMEM, "staging allocation failed");
        k_pack_writeback<<<(unsigned)((n + 255) / 256), 256, 0, s->stream>>>(s->pos, s->posc, s->vel, s->velc, s->acc,
                                                                            (int)n, 0, d_wb);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(h, d_wb, n * sizeof(WbRecord), cudaMemcpyDeviceToHost, s->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
        if (e != cudaSuccess) return cuda_fail(s, e, "nb_read_state");
        int rc = check_device_error(s);
        if (rc) return rc;
        for (size_t i = 0; i < n; ++i) {
            if (pos3) { pos3[3 * i] = h[i].pos[0]; pos3[3 * i + 1] = h[i].pos[1]; pos3[3 * i + 2] = h[i].pos[2]; }
            if (vel3) { vel3[3 * i] = h[i].vel[0]; vel3[3 * i + 1] = h[i].vel[1]; vel3[3 * i + 2] = h[i].vel[2]; }
            if (force3) { force3[3 * i] = h[i].force[0]; force3[3 * i + 1] = h[i].force[1]; force3[3 * i + 2] = h[i].force[2]; }
        }
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_write_back_direct(const nb_sim* s) {
    try {
     return s ? (host_direct(s) ? 1 : 0) : -1; 
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_write_back(nb_sim* s, nb_particle* particles, size_t n) {
    try {
        if (!s) return NB_EINVAL;
        if (n != s->n) return fail(s, NB_EINVAL, "record count differs from the initialised count");
        if (n == 0) return NB_OK;
        if (!particles) return fail(s, NB_EINVAL, "null particle buffer");
        cudaSetDevice(s->dev);
        const int zero = (s->prm.kind != NB_SIM_BARNES_HUT) && !s->forces_fresh;
        if (host_direct(s) && ((uintptr_t)particles & 3) == 0) {
            const size_t blocks = (n + 32 * kWbWarps - 1) / (32 * kWbWarps);
            cudaError_t e = nb::launch_after(
                k_writeback_records, (unsigned)std::min(blocks, (size_t)kWbPerSm * (size_t)s->sm_count), 32 * kWbWarps, 0,
                s->stream, s->pos, s->vel, s->velc, s->acc, (int)n, zero, reinterpret_cast<uint32_t*>(particles), s->d_err,
                s->h_err);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
            if (e != cudaSuccess) return cuda_fail(s, e, "nb_write_back");
            return decode_device_error(s);
        }
        WbRecord* d_wb = static_cast<WbRecord*>(device_stage(s, n * sizeof(WbRecord)));
        WbRecord* h_wb = static_cast<WbRecord*>(host_stage(s, n * sizeof(WbRecord)));
        if (!d_wb || !h_wb) return fail(s, NB_ENOMEM, "staging allocation failed");
        k_pack_writeback<<<(unsigned)((n + 255) / 256), 256, 0, s->stream>>>(s->pos, s->posc, s->vel, s->velc, s->acc,
                                                                            (int)n, zero, d_wb);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(h_wb, d_wb, n * sizeof(WbRecord), cudaMemcpyDeviceToHost, s->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(s->h_err, s->d_err, sizeof(int), cudaMemcpyDeviceToHost, s->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
        if (e != cudaSuccess) return cuda_fail(s, e, "nb_write_back");
        int rc = decode_device_error(s);
        if (rc) return rc;
        auto scatter = [&](size_t b, size_t end) {
            for (size_t i = b; i < end; ++i) {
                nb_particle& p = particles[i];
                const WbRecord& r = h_wb[i];
                p.position[0] = r.pos[0]; p.position[1] = r.pos[1]; p.position[2] = r.pos[2];
                p.velocity[0] = r.vel[0]; p.velocity[1] = r.vel[1]; p.velocity[2] = r.vel[2];
                p.forces[0] = r.force[0]; p.forces[1] = r.force[1]; p.forces[2] = r.force[2];
            }
        };
        const size_t kPar = 1 << 17;
        if (n >= 2 * kPar) {
            unsigned hc = std::max(2u, std::min(16u, std::thread::hardware_concurrency()));
            std::vector<std::thread> th;
            const size_t per = (n + hc - 1) / hc;
            for (unsigned t = 0; t < hc; ++t) {
                const size_t b = t * per, end = std::min(n, b + per);
                if (b < end) th.emplace_back(scatter, b, end);
            }
            for (auto& x : th) x.join();
        } else {
            scatter(0, n);
        }
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_compute_forces(nb_sim* s, double* force3) {
    try {
        if (!s) return NB_EINVAL;
        if (s->n == 0) return NB_OK;
        cudaSetDevice(s->dev);
        int rc = force_pass(s, 0.f, false);
        if (rc) return rc;
        if (!force3) return check_device_error(s);
        return nb_read_state(s, nullptr, nullptr, force3);
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_last_interactions(nb_sim* s, uint64_t* interactions) {
    try {
        if (!s || !interactions) return NB_EINVAL;
        cudaSetDevice(s->dev);
        if (s->prm.kind == NB_SIM_BARNES_HUT && s->tree.interactions) {
            unsigned long long v = 0;
            NB_CUDA(s, cudaMemcpyAsync(&v, s->tree.interactions, sizeof(v), cudaMemcpyDeviceToHost, s->stream));
            NB_CUDA(s, cudaStreamSynchronize(s->stream));
            s->inter_last = v;
        }
        *interactions = s->inter_last;
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_fp64_forces(nb_sim* s, const int32_t* targets, size_t m, double* force3) {
    try {
        if (!s) return NB_EINVAL;
        if (m == 0) return NB_OK;
        if (!targets || !force3) return fail(s, NB_EINVAL, "null buffer");
        for (size_t k = 0; k < m; ++k)
            if (targets[k] < 0 || (size_t)targets[k] >= s->n) return fail(s, NB_EINVAL, "target index out of range");
        cudaSetDevice(s->dev);
        int32_t* d_t = nullptr;
        double* d_o = nullptr;
        NB_CUDA(s, cudaMallocAsync(&d_t, m * sizeof(int32_t), s->stream));
        NB_CUDA(s, cudaMallocAsync(&d_o, m * 3 * sizeof(double), s->stream));
        cudaError_t e = cudaMemcpyAsync(d_t, targets, m * sizeof(int32_t), cudaMemcpyHostToDevice, s->stream);
        if (e == cudaSuccess) e = fp64_forces(s, d_t, m, d_o);
        if (e == cudaSuccess) e = cudaMemcpyAsync(force3, d_o, m * 3 * sizeof(double), cudaMemcpyDeviceToHost, s->stream);
        cudaFreeAsync(d_t, s->stream);
        cudaFreeAsync(d_o, s->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
        if (e != cudaSuccess) return cuda_fail(s, e, "nb_fp64_forces");
        return check_device_error(s);
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_diagnostics(nb_sim* s, float half_kick_dt, nb_diag* out) {
    try {
        if (!s || !out) return NB_EINVAL;
        std::memset(out, 0, sizeof(*out));
        if (s->n == 0) return NB_OK;
        cudaSetDevice(s->dev);
        if (half_kick_dt != 0.f) {
            int rc = force_pass(s, 0.f, false);   // acceleration at the current positions
            if (rc) return rc;
        }
        // the result goes through the handle's kept staging: an allocation a call
        // mapped and unmapped memory, about 100 us
        double* d_o = static_cast<double*>(device_stage(s, 12 * sizeof(double)));
        double* h = static_cast<double*>(host_stage(s, 12 * sizeof(double)));
        if (!d_o || !h) return fail(s, NB_ENOMEM, "staging allocation failed");
        cudaError_t e = fp64_diagnostics_ex(s, half_kick_dt, half_kick_dt != 0.f, true, d_o);
        if (e == cudaSuccess) e = cudaMemcpyAsync(h, d_o, 12 * sizeof(double), cudaMemcpyDeviceToHost, s->stream);
        if (e != cudaSuccess) return cuda_fail(s, e, "nb_diagnostics");
        const int rc = check_device_error(s);   // waits for the copies
        if (rc == NB_ECUDA) return rc;
        out->kinetic = h[0];
        out->potential = h[11];
        out->total = h[0] + h[11];
        out->momentum[0] = h[1]; out->momentum[1] = h[2]; out->momentum[2] = h[3];
        out->angular_momentum[0] = h[4]; out->angular_momentum[1] = h[5]; out->angular_momentum[2] = h[6];
        out->mass = h[7];
        for (int k = 0; k < 3; ++k) out->centre_of_mass[k] = h[7] != 0.0 ? h[8 + k] / h[7] : 0.0;
        return rc;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_render_vertices(nb_sim* s, const float* colour4, float scale, nb_render_vertex* out, size_t n) {
    try {
        if (!s || !out) return NB_EINVAL;
        if (n != s->n) return fail(s, NB_EINVAL, "vertex count differs from the initialised count");
        if (n == 0) return NB_OK;
        cudaSetDevice(s->dev);
        float4* d_c = nullptr;
        nb_render_vertex* d_v = nullptr;
        NB_CUDA(s, cudaMallocAsync(&d_v, n * sizeof(nb_render_vertex), s->stream));
        cudaError_t e = cudaSuccess;
        if (colour4) {
            e = cudaMallocAsync(&d_c, n * sizeof(float4), s->stream);
            if (e == cudaSuccess) e = cudaMemcpyAsync(d_c, colour4, n * sizeof(float4), cudaMemcpyHostToDevice, s->stream);
        }
        if (e == cudaSuccess) {
            k_render_fill<<<(unsigned)((n + 255) / 256), 256, 0, s->stream>>>(s->pos, d_c, scale, (int)n, d_v);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(out, d_v, n * sizeof(nb_render_vertex), cudaMemcpyDeviceToHost, s->stream);
        if (d_c) cudaFreeAsync(d_c, s->stream);
        cudaFreeAsync(d_v, s->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
        if (e != cudaSuccess) return cuda_fail(s, e, "nb_render_vertices");
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_render_attach(nb_sim* s, const float* colour4, float scale, void** device_vertices) {
    try {
        if (!s || !device_vertices) return NB_EINVAL;
        if (s->n == 0) return fail(s, NB_EBADSTATE, "nb_init_* first");
        cudaSetDevice(s->dev);
        detach_render(s);
        const size_t n = s->n;
        NB_CUDA(s, cudaMalloc(&s->render, n * sizeof(nb_render_vertex)));
        cudaError_t e = cudaMalloc(&s->rcolour, n * sizeof(float4));
        if (e == cudaSuccess) {
            if (colour4) {
                e = cudaMemcpyAsync(s->rcolour, colour4, n * sizeof(float4), cudaMemcpyHostToDevice, s->stream);
            } else {
                std::vector<float4> white(n, make_float4(1.f, 1.f, 1.f, 1.f));
                e = cudaMemcpyAsync(s->rcolour, white.data(), n * sizeof(float4), cudaMemcpyHostToDevice, s->stream);
                if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);   // before `white` goes away
            }
        }
        if (e == cudaSuccess) {
            s->rscale = scale;
            k_render_fill<<<(unsigned)((n + 255) / 256), 256, 0, s->stream>>>(s->pos, s->rcolour, scale, (int)n,
                                                                             s->render);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
        if (e != cudaSuccess) {
            detach_render(s);
            return cuda_fail(s, e, "nb_render_attach");
        }
        *device_vertices = s->render;
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_render_detach(nb_sim* s) {
    try {
        if (!s) return NB_EINVAL;
        cudaSetDevice(s->dev);
        cudaStreamSynchronize(s->stream);
        detach_render(s);
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_render_read(nb_sim* s, nb_render_vertex* out, size_t n) {
    try {
        if (!s || (!out && n)) return NB_EINVAL;
        if (!s->render) return fail(s, NB_EBADSTATE, "no vertex buffer attached");
        if (n != s->n) return fail(s, NB_EINVAL, "vertex count differs from the initialised count");
        cudaSetDevice(s->dev);
        NB_CUDA(s, cudaMemcpyAsync(out, s->render, n * sizeof(nb_render_vertex), cudaMemcpyDeviceToHost, s->stream));
        NB_CUDA(s, cudaStreamSynchronize(s->stream));
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

}  // extern "C"

// ---- profiling ---------------------------------------------------------------
namespace nb {

static cudaEvent_t take_event(nb_sim* s) {
    if (!s->prof.pool.empty()) {
        cudaEvent_t e = s->prof.pool.back();
        s->prof.pool.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    if (cudaEventCreate(&e) != cudaSuccess) return nullptr;
    return e;
}

static void drain_profile(nb_sim* s) {
    if (s->prof.pending.empty()) return;
    cudaStreamSynchronize(s->stream);
    for (auto& p : s->prof.pending) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, p.a, p.b) == cudaSuccess) {
            s->prof.ms[p.phase] += ms;
            s->prof.count[p.phase] += 1;
        }
        s->prof.pool.push_back(p.a);
        s->prof.pool.push_back(p.b);
    }
    s->prof.pending.clear();
    cudaGetLastError();
}

PhaseScope::PhaseScope(nb_sim* sim, int phase, int launches) : sim_(sim), phase_(phase) {
    sim_->prof.launches += (uint64_t)launches;
    if (!sim_->prof.on) return;
    if (sim_->prof.pending.size() > 4096) drain_profile(sim_);
    cudaEvent_t a = take_event(sim_);
    b_ = take_event(sim_);
    if (!a || !b_) { b_ = nullptr; return; }
    cudaEventRecord(a, sim_->stream);
    sim_->prof.pending.push_back({phase_, a, b_});
}

PhaseScope::~PhaseScope() {
    if (b_) cudaEventRecord(b_, sim_->stream);
}

__global__ void k_fma_probe(float* out, int iters, float a, float b) {
    float x0 = threadIdx.x * 1e-3f, x1 = x0 + 1.f, x2 = x0 + 2.f, x3 = x0 + 3.f;
    float x4 = x0 + 4.f, x5 = x0 + 5.f, x6 = x0 + 6.f, x7 = x0 + 7.f;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            x0 = fmaf(x0, a, b); x1 = fmaf(x1, a, b); x2 = fmaf(x2, a, b); x3 = fmaf(x3, a, b);
            x4 = fmaf(x4, a, b); x5 = fmaf(x5, a, b); x6 = fmaf(x6, a, b); x7 = fmaf(x7, a, b);
        }
    }
    const float r = ((x0 + x1) + (x2 + x3)) + ((x4 + x5) + (x6 + x7));
    if (r == 1234.5678f) out[0] = r;   // keeps the chains alive
}

}  // namespace nb

extern "C" {

int nb_profile_enable(nb_sim* s, int on) {
    try {
        if (!s) return NB_EINVAL;
        cudaSetDevice(s->dev);
        nb::drain_profile(s);
        s->prof.on = on != 0;
        if (on) {
            for (int k = 0; k < nb::kPhases; ++k) { s->prof.ms[k] = 0.0; s->prof.count[k] = 0; }
        }
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_profile_read(nb_sim* s, int phase, double* total_ms, uint64_t* launches) {
    try {
        if (!s || phase < 0 || phase >= nb::kPhases) return NB_EINVAL;
        cudaSetDevice(s->dev);
        nb::drain_profile(s);
        if (total_ms) *total_ms = s->prof.ms[phase];
        if (launches) *launches = s->prof.count[phase];
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_launch_count(nb_sim* s, uint64_t* launches) {
    try {
        if (!s || !launches) return NB_EINVAL;
        *launches = s->prof.launches;
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_probe_fp32_peak(int device, double* tflops) {
    try {
        if (!tflops) return NB_EINVAL;
        *tflops = 0.0;
        if (cudaSetDevice(device) != cudaSuccess) { cudaGetLastError(); return NB_ECUDA; }
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        float* d = nullptr;
        if (cudaMalloc(&d, sizeof(float)) != cudaSuccess) { cudaGetLastError(); return NB_ECUDA; }
        cudaEvent_t a, b;
        cudaEventCreate(&a);
        cudaEventCreate(&b);
        const int threads = 512, blocks = sms * 4, iters = 4096;
        nb::k_fma_probe<<<blocks, threads>>>(d, 64, 1.0000001f, 1e-7f);   // warm-up
        cudaEventRecord(a);
        nb::k_fma_probe<<<blocks, threads>>>(d, iters, 1.0000001f, 1e-7f);
        cudaEventRecord(b);
        cudaError_t e = cudaEventSynchronize(b);
        float ms = 0.f;
        if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, a, b);
        cudaEventDestroy(a);
        cudaEventDestroy(b);
        cudaFree(d);
        if (e != cudaSuccess || ms <= 0.f) { cudaGetLastError(); return NB_ECUDA; }
        const double flops = 2.0 * 8.0 * 16.0 * (double)iters * (double)threads * (double)blocks;
        *tflops = flops / (ms * 1e-3) / 1e12;
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

}  // extern "C"

extern "C" {

int nb_tune(nb_sim* s, const char* key, int value) {
    try {
        if (!s || !key) return NB_EINVAL;
        const std::string k(key);
        if (k == "direct_block") {
            if (value != 64 && value != 128 && value != 256) return NB_EINVAL;
            s->tune.block = value;
        } else if (k == "direct_ipt") {
            if (value != 1 && value != 2 && value != 4 && value != 8) return NB_EINVAL;
            if (value == 8 && s->tune.block == 256) return NB_EINVAL;
            s->tune.ipt = value;
        } else if (k == "direct_splits") {
            if (value < 0 || value > 4096) return NB_EINVAL;
            s->tune.splits = value;
        } else if (k == "wait_polls") {
            if (value < 0 || value > (int)nb::kMaxPolls) return NB_EINVAL;
            s->wait_polls = (uint32_t)value;
            return NB_OK;
        } else {
            return NB_EINVAL;
        }
        s->tune_set = true;
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

int nb_get_tune(nb_sim* s, const char* key, int* value) {
    try {
        if (!s || !key || !value) return NB_EINVAL;
        const std::string k(key);
        if (k == "direct_block") *value = s->tune.block;
        else if (k == "direct_ipt") *value = s->tune.ipt;
        else if (k == "direct_splits") *value = s->tune.splits;
        else if (k == "wait_polls") *value = (int)s->wait_polls;
        else return NB_EINVAL;
        return NB_OK;
    } catch (...) {   // no exception crosses the C-ABI: host allocation failed
        return NB_ENOMEM;
    }
}

}  // extern "C"

namespace nb {

__global__ void k_fma2_probe(float* out, int iters, float a, float b) {
    const float2 A = make_float2(a, a), B = make_float2(b, b);
    float2 x0 = make_float2(threadIdx.x * 1e-3f, 1.f), x1 = make_float2(2.f, 3.f), x2 = make_float2(4.f, 5.f);
    float2 x3 = make_float2(6.f, 7.f), x4 = make_float2(8.f, 9.f), x5 = make_float2(10.f, 11.f);
    float2 x6 = make_float2(12.f, 13.f), x7 = make_float2(14.f, 15.f);
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            x0 = __ffma2_rn(x0, A, B); x1 = __ffma2_rn(x1, A, B); x2 = __ffma2_rn(x2, A, B); x3 = __ffma2_rn(x3, A, B);
            x4 = __ffma2_rn(x4, A, B); x5 = __ffma2_rn(x5, A, B); x6 = __ffma2_rn(x6, A, B); x7 = __ffma2_rn(x7, A, B);
        }
    }
    const float r = ((x0.x + x1.x) + (x2.x + x3.x)) + ((x4.y + x5.y) + (x6.y + x7.y));
    if (r == 1234.5678f) out[0] = r;
}

}  // namespace nb

extern "C" int nb_probe_fp32x2_peak(int device, double* tflops) {
    if (!tflops) return NB_EINVAL;
    *tflops = 0.0;
    if (cudaSetDevice(device) != cudaSuccess) { cudaGetLastError(); return NB_ECUDA; }
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    float* d = nullptr;
    if (cudaMalloc(&d, sizeof(float)) != cudaSuccess) { cudaGetLastError(); return NB_ECUDA; }
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    const int threads = 512, blocks = sms * 4, iters = 4096;
    nb::k_fma2_probe<<<blocks, threads>>>(d, 64, 1.0000001f, 1e-7f);
    cudaEventRecord(a);
    nb::k_fma2_probe<<<blocks, threads>>>(d, iters, 1.0000001f, 1e-7f);
    cudaEventRecord(b);
    cudaError_t e = cudaEventSynchronize(b);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(d);
    if (e != cudaSuccess || ms <= 0.f) { cudaGetLastError(); return NB_ECUDA; }
    // 2 lanes x 2 flops per FFMA2
    const double flops = 4.0 * 8.0 * 16.0 * (double)iters * (double)threads * (double)blocks;
    *tflops = flops / (ms * 1e-3) / 1e12;
    return NB_OK;
}
