// k_direct.cu -- all-pairs kernels: the direct sums (update /
// update_local, kernels/brute_force_update.cl) and copy_vertices
// (kernels/copy_vertices.cl), plus the host-layout pack/unpack kernels.
//
// The direct sums are direct_device.cuh's; this file splits them over the GPU.
#include <algorithm>

#include "direct_device.cuh"
#include "integrate.cuh"
#include "launch.cuh"

namespace nbgb {

// ---------------------------------------------------------------------------
// One block: 32 kI targets (blockIdx.x) over one of gridDim.y slices of the
// bodies.  With one slice the block integrates its targets; with more it
// writes its sums to part[slice][target], and the block that finishes a
// target set last adds the slices in order and integrates: one launch, no
// atomics on the sums, the same bits every time.  `arrived` counts the blocks
// of each set that are done; the last one puts it back to zero.
// out (allocation-free form): accelerations instead of the integrator.
// ---------------------------------------------------------------------------
constexpr int kDirectWarps = kDirectStreams;
template <int kI, bool kQuirk, int kZero>
__global__ void __launch_bounds__(32 * kDirectWarps, kI == 4 ? 2 : 3)
    k_direct(DevSim s, StepParams p, float4 *part, int *arrived, float4 *out) {
    wait_for_previous();
    __shared__ DirectShared<kI, kDirectWarps> sh;
    __shared__ int last;
    const int n = s.n, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int base = blockIdx.x * (32 * kI);
    // slices of whole tiles
    const int tiles = (n + kDirectTile - 1) / kDirectTile;
    const int per = (tiles + gridDim.y - 1) / gridDim.y * kDirectTile;
    const int j0 = blockIdx.y * per, j1 = min(n, j0 + per);
    direct_sum<kI, kDirectWarps, kQuirk, kZero>(s.body_cur, n, j0, j1, base, p.eps, warp, lane, sh);
    float3 a = make_float3(0.0f, 0.0f, 0.0f);
    if (threadIdx.x < 32 * kI) a = direct_target_sum<kI, kDirectWarps>(sh, threadIdx.x);
    const int i = base + (int)threadIdx.x;
    const bool mine = threadIdx.x < 32 * kI && i < n;
    if (gridDim.y > 1) {
        if (mine) part[(size_t)blockIdx.y * n + i] = make_float4(a.x, a.y, a.z, 0.0f);
        __threadfence();  // the sums before the arrival
        __syncthreads();
        if (threadIdx.x == 0) last = atomicAdd(&arrived[blockIdx.x], 1) == (int)gridDim.y - 1;
        __syncthreads();
        if (!last) return;
        __threadfence();
        if (threadIdx.x == 0) arrived[blockIdx.x] = 0;
        if (mine) {
            a = make_float3(0.0f, 0.0f, 0.0f);
            for (int k = 0; k < (int)gridDim.y; ++k) {
                const float4 v = __ldcg(&part[(size_t)k * n + i]);
                a.x += v.x;
                a.y += v.y;
                a.z += v.z;
            }
        }
    }
    if (!mine) return;
    if (out) out[i] = make_float4(a.x * p.G, a.y * p.G, a.z * p.G, 0.0f);
    else integrate_any(s, p, i, s.body_cur[i], a.x * p.G, a.y * p.G, a.z * p.G);
}

__global__ void k_copy_vertices(const float4 *__restrict__ b, int n, float4 *__restrict__ dst) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 p = b[i];
        dst[i] = make_float4(p.x, p.y, p.z, 1.0f);
    }
}

// The reference's packed float[3N] arrays <-> the float4 body layout.  A
// block moves tiles of kPackTile bodies; when the float[3N] arrays are 16-byte
// aligned, a whole tile's 3 * kPackTile floats move as contiguous float4
// loads or stores through shared memory (the arrays may be host memory the
// device reads or writes directly, where full-width accesses matter),
// otherwise as one float at a time.
constexpr int kPackTile = 256;
constexpr int kPackVec = kPackTile * 3 / 4;  // float4 per tile of float[3]

__global__ void __launch_bounds__(kPackTile) k_pack(const float *__restrict__ pos3, const float *__restrict__ mass,
                                                    const float *__restrict__ vel3, float4 *body, float4 *vel,
                                                    float4 *acc, int n, int vec) {
    __shared__ float4 tp[kPackVec], tv[kPackVec];
    const float *fp = reinterpret_cast<const float *>(tp), *fv = reinterpret_cast<const float *>(tv);
    const int t = threadIdx.x;
    const int ntiles = (n + kPackTile - 1) / kPackTile;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const size_t i0 = (size_t)tile * kPackTile;
        const size_t i = i0 + t;
        const bool full = vec && i0 + kPackTile <= (size_t)n;  // block-uniform
        if (full && t < kPackVec) {
            if (pos3) tp[t] = reinterpret_cast<const float4 *>(pos3 + 3 * i0)[t];
            if (vel3) tv[t] = reinterpret_cast<const float4 *>(vel3 + 3 * i0)[t];
        }
        __syncthreads();
        if (i < (size_t)n) {
            if (pos3) {
                const float m = mass ? mass[i] : body[i].w;
                body[i] = full ? make_float4(fp[3 * t], fp[3 * t + 1], fp[3 * t + 2], m)
                               : make_float4(pos3[3 * i], pos3[3 * i + 1], pos3[3 * i + 2], m);
            } else if (mass) {
                body[i].w = mass[i];
            }
            if (vel) {
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (vel3) v = full ? make_float4(fv[3 * t], fv[3 * t + 1], fv[3 * t + 2], 0.0f)
                                   : make_float4(vel3[3 * i], vel3[3 * i + 1], vel3[3 * i + 2], 0.0f);
                vel[i] = v;
            }
            if (acc) acc[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        __syncthreads();  // the tile is read before the next one is staged
    }
}

// one float4 array -> one float[3N] array, tile at i0 (block-uniform `full`)
__device__ __forceinline__ void unpack_tile(const float4 *__restrict__ src, float *dst, size_t i0, int n, bool full,
                                            float4 *tile) {
    const int t = threadIdx.x;
    const size_t i = i0 + t;
    if (full) {
        float *f = reinterpret_cast<float *>(tile);
        const float4 v = src[i];
        f[3 * t] = v.x;
        f[3 * t + 1] = v.y;
        f[3 * t + 2] = v.z;
        __syncthreads();
        if (t < kPackVec) reinterpret_cast<float4 *>(dst + 3 * i0)[t] = tile[t];
        __syncthreads();
    } else if (i < (size_t)n) {
        const float4 v = src[i];
        dst[3 * i] = v.x;
        dst[3 * i + 1] = v.y;
        dst[3 * i + 2] = v.z;
    }
}

__global__ void __launch_bounds__(kPackTile) k_unpack(const float4 *__restrict__ body, const float4 *__restrict__ vel,
                                                      const float4 *__restrict__ acc, float *pos3, float *vel3,
                                                      float *acc3, float *mass, int n, int vec) {
    __shared__ float4 tile[kPackVec];
    const int ntiles = (n + kPackTile - 1) / kPackTile;
    for (int k = blockIdx.x; k < ntiles; k += gridDim.x) {
        const size_t i0 = (size_t)k * kPackTile;
        const bool full = vec && i0 + kPackTile <= (size_t)n;  // block-uniform
        if (pos3) unpack_tile(body, pos3, i0, n, full, tile);
        if (vel3) unpack_tile(vel, vel3, i0, n, full, tile);
        if (acc3) unpack_tile(acc, acc3, i0, n, full, tile);
        if (mass && i0 + threadIdx.x < (size_t)n) mass[i0 + threadIdx.x] = body[i0 + threadIdx.x].w;
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
// Targets per lane and slices of the bodies: the pair that a model of the
// busiest SM finds fastest.  A block costs its tiles (64 bodies against 32 kI
// targets, divided over the warps), a pair somewhat more at small kI, plus a
// fixed part; an SM with one block is not kept busy by its eight warps; slices
// cost the exchange of their sums.  In units of one round of tiles of 32
// targets.  Fitted to every (kI, slices) timed on a GB300 at twelve sizes; what
// it takes is within 1 % of the best of them from 8,192 bodies up (20,000: kI =
// 2, 10 slices 160 us, best 158, one slice of kI = 4 252; 262,144: kI = 4 24.65
// ms, kI = 2 24.91, kI = 1 26.57) and within one launch quantum (2 us) below.
DirectPlan direct_plan(int n, int sm_count, int max_slices) {
    static const float kPair[3] = {1.05f, 1.02f, 1.0f};  // kI = 1, 2, 4
    const int tiles = (n + kDirectTile - 1) / kDirectTile;
    DirectPlan best{1, 1};
    float best_cost = 0.0f;
    for (int v = 0; v < 3; ++v) {
        const int ki = 1 << v;
        const long long sets = ((long long)n + 32 * ki - 1) / (32 * ki);
        for (int slices = 1; slices <= max_slices; ++slices) {
            const int per = (tiles + slices - 1) / slices;  // tiles a block
            if (slices > 1 && (long long)(slices - 1) * per >= tiles) continue;  // an empty slice
            const long long on_sm = (sets * slices + sm_count - 1) / sm_count;
            const float sum = (float)((per + kDirectWarps - 1) / kDirectWarps) * ki * kPair[v];
            const float cost = (float)on_sm * (sum * (on_sm == 1 ? 1.4f : 1.0f) + 0.3f) + (slices > 1 ? 2.0f : 0.0f);
            if (best_cost == 0.0f || cost < best_cost) {
                best_cost = cost;
                best = DirectPlan{ki, slices};
            }
        }
    }
    return best;
}

template <bool kQuirk, int kZero>
static cudaError_t launch_direct_z(const DevSim &s, const StepParams &p, const DirectPlan &d, float4 *part,
                                   int *arrived, float4 *out, cudaStream_t st) {
    const dim3 grid((unsigned)((s.n + 32 * d.ki - 1) / (32 * d.ki)), (unsigned)d.slices);
    const int threads = 32 * kDirectWarps;
    return launch_next(d.ki == 4   ? k_direct<4, kQuirk, kZero>
                       : d.ki == 2 ? k_direct<2, kQuirk, kZero>
                                   : k_direct<1, kQuirk, kZero>,
                       grid, threads, st, s, p, part, arrived, out);
}

// `p.eps` is the softening to use; s.part (direct_part_bodies float4) holds
// the sums of the slices.
cudaError_t launch_direct(const DevSim &s, const StepParams &p, const DirectPlan &plan, int *arrived, int tiled,
                          int quirk, cudaStream_t st) {
    if (quirk) return launch_direct_z<true, kZeroAdds>(s, p, plan, s.part, arrived, nullptr, st);
    if (p.eps > 0.0f) return launch_direct_z<false, kZeroAdds>(s, p, plan, s.part, arrived, nullptr, st);
    if (tiled) return launch_direct_z<false, kZeroSkips>(s, p, plan, s.part, arrived, nullptr, st);
    return launch_direct_z<false, kZeroSkipsSelf>(s, p, plan, s.part, arrived, nullptr, st);
}

cudaError_t launch_copy_vertices(const float4 *body, int n, float4 *dst, cudaStream_t st) {
    k_copy_vertices<<<(n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096, 256, 0, st>>>(body, n, dst);
    return cudaGetLastError();
}

static bool aligned16(const void *p) { return ((uintptr_t)p & 15) == 0; }

cudaError_t launch_pack(const float *pos3, const float *mass, const float *vel3, float4 *body, float4 *vel,
                        float4 *acc, int n, cudaStream_t st) {
    const int tiles = (n + kPackTile - 1) / kPackTile;
    const int blocks = tiles < 4096 ? tiles : 4096;
    const int vec = aligned16(pos3) && aligned16(vel3);
    k_pack<<<blocks > 0 ? blocks : 1, kPackTile, 0, st>>>(pos3, mass, vel3, body, vel, acc, n, vec);
    return cudaGetLastError();
}

cudaError_t launch_unpack(const float4 *body, const float4 *vel, const float4 *acc, float *pos3, float *vel3,
                          float *acc3, float *mass, int n, cudaStream_t st) {
    const int tiles = (n + kPackTile - 1) / kPackTile;
    const int blocks = tiles < 4096 ? tiles : 4096;
    const int vec = aligned16(pos3) && aligned16(vel3) && aligned16(acc3);
    k_unpack<<<blocks > 0 ? blocks : 1, kPackTile, 0, st>>>(body, vel, acc, pos3, vel3, acc3, mass, n, vec);
    return cudaGetLastError();
}

}  // namespace nbgb

namespace nbgb {

// ===========================================================================
// Allocation-free all-pairs accelerations (nb_direct_accel_noalloc).
//
// For callers that must not allocate device memory: a host engine that owns
// the whole device-memory budget and hands the library only its own buffers,
// or a frame loop where a cudaMalloc (which can synchronise the device and
// take an allocator lock) is not allowed.  The caller passes the bodies and
// the output; the one piece of scratch the split all-pairs sum needs -- the
// partial accelerations of the body slices -- lives in a file-scope device
// array of fixed size, together with the counters of the slices that are
// done.  Every GPU that loads this library holds that array (1 MiB + 8 KiB)
// until the process exits.  All calls share it: calls that overlap on the GPU
// race, and only they: the counters they may leave behind are cleared by the next
// call that has the array to itself (NoAllocCall).
// ===========================================================================
constexpr int kNoAllocMaxBodies = 65536;  // = NB_NOALLOC_MAX_BODIES
static __device__ __align__(256) float4 g_noalloc_part[kNoAllocMaxBodies];
static __device__ __align__(256) int g_noalloc_arrived[kNoAllocMaxBodies / 32];

}  // namespace nbgb

#include <mutex>

#include "../../include/nbgb.h"

static_assert(nbgb::kNoAllocMaxBodies == NB_NOALLOC_MAX_BODIES, "the scratch must hold the documented limit");

namespace {
// Device addresses of the two arrays, looked up once per device with that
// device current.  In host code the array names are host-side stand-ins, not
// device addresses, so only these looked-up pointers are passed to kernels.
// The addresses are kept for the life of the process: a cudaDeviceReset (or
// a reset of the device's primary context) unloads the module, after which
// this entry point must not be called on that device again.
constexpr int kMaxDevices = 64;
struct NoAllocDevice {
    void *part = nullptr, *arrived = nullptr;
    int calls = 0;         // between their first launch and the end of their synchronisation
    bool unclean = false;  // calls overlapped, or one failed: its counters may not be zero
};
std::mutex g_noalloc_mu;
NoAllocDevice g_noalloc_dev[kMaxDevices];

// One call's turn on the shared array.  A call that meets no other finds the
// counters at zero, as its own last blocks leave them, or clears them first.
class NoAllocCall {
  public:
    explicit NoAllocCall(int dev) : d_(g_noalloc_dev[dev]) {
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!d_.part) {
            void *p = nullptr, *c = nullptr;
            if (cudaGetSymbolAddress(&p, nbgb::g_noalloc_part) != cudaSuccess) return;
            if (cudaGetSymbolAddress(&c, nbgb::g_noalloc_arrived) != cudaSuccess) return;
            d_.part = p;
            d_.arrived = c;
        }
        ok_ = true;
        if (d_.calls++ > 0) d_.unclean = true;
        clear_ = d_.unclean && d_.calls == 1;
        if (clear_) d_.unclean = false;
    }
    ~NoAllocCall() {
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!ok_) return;
        --d_.calls;
        if (!done_) d_.unclean = true;
    }
    bool ok() const { return ok_; }
    bool clear() const { return clear_; }
    float4 *part() const { return static_cast<float4 *>(d_.part); }
    int *arrived() const { return static_cast<int *>(d_.arrived); }
    void done() { done_ = true; }

  private:
    NoAllocDevice &d_;
    bool ok_ = false, clear_ = false, done_ = false;
};
}  // namespace

extern "C" nb_status nb_direct_accel_noalloc(const float *d_body4, int32_t n, float eps, float G, float *d_acc4,
                                            void *stream) {
    using namespace nbgb;
    if (!d_body4 || !d_acc4 || n < 1 || !(eps >= 0.0f)) return NB_ERR_INVALID_ARGUMENT;
    if (n > kNoAllocMaxBodies) return NB_ERR_INVALID_ARGUMENT;  // beyond the fixed scratch
    if (((uintptr_t)d_body4 & 15u) || ((uintptr_t)d_acc4 & 15u)) return NB_ERR_INVALID_ARGUMENT;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return NB_ERR_NO_DEVICE;
    NoAllocCall call(dev);
    if (!call.ok()) return NB_ERR_CUDA;
    float4 *part = call.part();
    int *arrived = call.arrived();
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (call.clear() && cudaMemsetAsync(arrived, 0, sizeof(int) * (kNoAllocMaxBodies / 32), st) != cudaSuccess)
        return NB_ERR_CUDA;
    int sm_count = 0;
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
    DevSim s{};
    s.n = n;
    s.body_cur = reinterpret_cast<const float4 *>(d_body4);
    StepParams p{};
    p.eps = eps;
    p.G = G;
    float4 *out = reinterpret_cast<float4 *>(d_acc4);
    // the caller may have the accelerations written over the bodies: then
    // they go through the scratch, in one slice
    const uintptr_t b0 = (uintptr_t)d_body4, a0 = (uintptr_t)d_acc4, bytes = sizeof(float4) * (size_t)n;
    const bool overlap = a0 < b0 + bytes && b0 < a0 + bytes;
    const DirectPlan plan = direct_plan(n, sm_count, overlap ? 1 : std::min(kDirectMaxSlices, kNoAllocMaxBodies / n));
    if (overlap) out = part;
    const cudaError_t e = eps > 0.0f ? launch_direct_z<false, kZeroAdds>(s, p, plan, part, arrived, out, st)
                                     : launch_direct_z<false, kZeroSkips>(s, p, plan, part, arrived, out, st);
    if (e != cudaSuccess) return NB_ERR_CUDA;
    if (overlap && cudaMemcpyAsync(d_acc4, part, bytes, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
        return NB_ERR_CUDA;
    if (cudaStreamSynchronize(st) != cudaSuccess) return NB_ERR_CUDA;
    call.done();
    return NB_OK;
}
