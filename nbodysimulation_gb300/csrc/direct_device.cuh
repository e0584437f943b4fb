// direct_device.cuh -- the all-pairs sum of one block (update / update_local,
// kernels/brute_force_update.cl), shared by the single-system and
// allocation-free kernels (k_direct.cu) and the batched one (k_batch.cu).
//
// A block of kW warps sums 32 kI targets over the bodies [j0, j1).  The bodies'
// tiles of 64 are dealt to eight streams, whatever kW and kI are, so a target's sum
// depends on the bodies alone: no shape of a batch's kernel changes a result.
// Every warp has all the targets (kI per lane, in registers for the whole sum) and
// sums its streams one after another, at its own pace -- no block barrier until the
// streams' sums are added, in their order, at the end.  A lane loads two
// consecutive bodies of the next tile while the warp sums this one, and stores
// them as a pair {x0,x1,y0,y1}, {z0,z1,m0,m1}: what the packed FP32
// instructions take, so one pair of broadcast loads feeds 2 kI interactions
// per lane.  The bodies pass through registers on their way to that form, which
// is why they are loaded and not brought by bulk copies.
//
// Bound by the FP32 arithmetic and its register reads: 12 operations and one
// MUFU a pair, 14.4 issue cycles a warp at kI = 4 (16 scalar operations, four
// targets and tiles brought by bulk copies took 17.2).  Whole steps on a GB300,
// against that kernel with its separate clearing and integrating launches for
// small systems: 262,144 bodies 29.4 -> 24.7 ms (2.78e12 pairs/s, 83 % of the
// FP32 lanes), 50,021 1.53 -> 0.93 ms, 20,000 0.336 -> 0.160 ms, 4,096 27 -> 14
// us; the direct half of a batch (30 systems of 1,043 to 8,139 bodies) 0.55 ->
// 0.19 ms.
#pragma once
#include "packed.cuh"

namespace nbgb {

constexpr int kDirectTile = 64;   // bodies per tile of one warp: two per lane
constexpr int kDirectStreams = 8;  // stream w: tiles w, w + 8, ...
// how a pair at zero distance counts
enum { kZeroAdds = 0,      // eps > 0: nothing special
       kZeroSkips = 1,     // eps = 0, update_local's form: adds nothing
       kZeroSkipsSelf = 2  // eps = 0, update's form: only the body itself is skipped
};

template <int kI>
struct DirectTargets {
    float2 nx[kI], ny[kI], nz[kI];  // minus the positions, twice
    float2 ax[kI], ay[kI], az[kI];  // sums over the even and the odd bodies
};

template <int kI, int kW>
struct __align__(16) DirectShared {
    static_assert(kDirectStreams % kW == 0, "every warp has as many streams");
    static constexpr bool kOver = kW == kDirectStreams;  // the streams' sums lie where the tiles were
    static constexpr int kSums = (3 * kI * kDirectStreams * 32 * 4 + 2047) / 2048;  // in warps' tiles
    static_assert(!kOver || kW >= kSums, "the sums fit in the tiles' memory");
    float4 tile[kOver ? kW : kW + kSums][2][kDirectTile];  // per warp, double-buffered: 32 x {x0,x1,y0,y1}, 32 x {z0,z1,m0,m1}
    __device__ __forceinline__ float *sums() { return reinterpret_cast<float *>(tile[kOver ? 0 : kW]); }  // [stream][component][target]
};

// the reference's brute-force arithmetic: n = normalize(r), s = m / (|n|^2 +
// e^2) (brute_force_update.cl:54-60, 114-123); the zero vector normalises to
// zero, so the self pair adds nothing
__device__ __forceinline__ void quirk_pair(float dx, float dy, float dz, float m, float eps2, float &ax, float &ay,
                                           float &az) {
    const float l2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    const float inv = l2 > 0.0f ? rsqrtf(l2) : 0.0f;
    const float nx = dx * inv, ny = dy * inv, nz = dz * inv;
    const float s = __fdividef(m, fmaf(nz, nz, fmaf(ny, ny, fmaf(nx, nx, eps2))));
    ax = fmaf(nx, s, ax);
    ay = fmaf(ny, s, ay);
    az = fmaf(nz, s, az);
}

// One stream of [j0, j1).  i0: index of the lane's first target, its others 32
// apart (kZeroSkipsSelf); buffers: the warp's two tiles.
template <int kI, bool kQuirk, int kZero>
__device__ __forceinline__ void direct_stream(const float4 *body, int j0, int j1, int i0, float eps, int stream,
                                              int lane, float4 (*buffers)[kDirectTile], DirectTargets<kI> &T) {
    const float2 eps2 = dup(eps * eps);
    const int tiles = (j1 - j0 + kDirectTile - 1) / kDirectTile;
    float4 p0, p1;
    // bodies beyond the range: the range's last one without mass
    auto load = [&](int t) {
        const int j = j0 + t * kDirectTile + 2 * lane;
        p0 = body[min(j, j1 - 1)];
        p1 = body[min(j + 1, j1 - 1)];
        if (j >= j1) p0.w = 0.0f;
        if (j + 1 >= j1) p1.w = 0.0f;
    };
    if (stream < tiles) load(stream);
    int buf = 0;
    for (int t = stream; t < tiles; t += kDirectStreams) {
        float4 *tl = buffers[buf];
        buf ^= 1;
        tl[lane] = make_float4(p0.x, p1.x, p0.y, p1.y);
        tl[32 + lane] = make_float4(p0.z, p1.z, p0.w, p1.w);
        __syncwarp();  // also: the tile before last is no longer read
        if (t + kDirectStreams < tiles) load(t + kDirectStreams);
#pragma unroll 4
        for (int k = 0; k < kDirectTile / 2; ++k) {
            const float4 xy = tl[k], zm = tl[32 + k];
            const float2 qx = lo2(xy), qy = hi2(xy), qz = lo2(zm), m = hi2(zm);
#pragma unroll
            for (int r = 0; r < kI; ++r) {
                const float2 dx = __fadd2_rn(qx, T.nx[r]), dy = __fadd2_rn(qy, T.ny[r]), dz = __fadd2_rn(qz, T.nz[r]);
                if constexpr (kQuirk) {
                    quirk_pair(dx.x, dy.x, dz.x, m.x, eps2.x, T.ax[r].x, T.ay[r].x, T.az[r].x);
                    quirk_pair(dx.y, dy.y, dz.y, m.y, eps2.y, T.ax[r].y, T.ay[r].y, T.az[r].y);
                } else {
                    const float2 d2 = pair_dist2(dx, dy, dz, eps2);
                    const float2 f = make_float2(rsqrt_fast(d2.x), rsqrt_fast(d2.y));
                    float2 F = __fmul2_rn(__fmul2_rn(m, f), __fmul2_rn(f, f));
                    if constexpr (kZero == kZeroSkips) {
                        F.x = d2.x > 0.0f ? F.x : 0.0f;
                        F.y = d2.y > 0.0f ? F.y : 0.0f;
                    }
                    if constexpr (kZero == kZeroSkipsSelf) {
                        const int j = j0 + t * kDirectTile + 2 * k;
                        if (j == i0 + 32 * r || j >= j1) F.x = 0.0f;
                        if (j + 1 == i0 + 32 * r || j + 1 >= j1) F.y = 0.0f;
                    }
                    T.ax[r] = __ffma2_rn(dx, F, T.ax[r]);
                    T.ay[r] = __ffma2_rn(dy, F, T.ay[r]);
                    T.az[r] = __ffma2_rn(dz, F, T.az[r]);
                }
            }
        }
    }
}

template <int kI>
__device__ __forceinline__ void direct_load_targets(const float4 *body, int i0, int n, DirectTargets<kI> &T) {
#pragma unroll
    for (int r = 0; r < kI; ++r) {
        const float4 P = body[min(i0 + 32 * r, n - 1)];
        T.nx[r] = dup(-P.x);
        T.ny[r] = dup(-P.y);
        T.nz[r] = dup(-P.z);
        T.ax[r] = T.ay[r] = T.az[r] = make_float2(0.0f, 0.0f);
    }
}

// The streams' sums of the block's targets (the first one `base`).  Every thread
// of the block calls it.
template <int kI, int kW, bool kQuirk, int kZero>
__device__ __forceinline__ void direct_sum(const float4 *body, int n, int j0, int j1, int base, float eps, int warp,
                                           int lane, DirectShared<kI, kW> &sh) {
    const int i0 = base + lane;
    DirectTargets<kI> T;
    direct_load_targets<kI>(body, i0, n, T);
    const auto store = [&](int stream) {
#pragma unroll
        for (int r = 0; r < kI; ++r) {
            float *at = sh.sums() + stream * (3 * 32 * kI) + 32 * r + lane;
            at[0] = T.ax[r].x + T.ax[r].y;
            at[32 * kI] = T.ay[r].x + T.ay[r].y;
            at[64 * kI] = T.az[r].x + T.az[r].y;
        }
    };
    if constexpr (DirectShared<kI, kW>::kOver) {
        direct_stream<kI, kQuirk, kZero>(body, j0, j1, i0, eps, warp, lane, sh.tile[warp], T);
        __syncthreads();  // the tiles are no longer read
        store(warp);
    } else {
        for (int stream = warp; stream < kDirectStreams; stream += kW) {
            direct_stream<kI, kQuirk, kZero>(body, j0, j1, i0, eps, stream, lane, sh.tile[warp], T);
            store(stream);
#pragma unroll
            for (int r = 0; r < kI; ++r) T.ax[r] = T.ay[r] = T.az[r] = make_float2(0.0f, 0.0f);
            __syncwarp();  // the next stream's tiles go where this one's were read
        }
    }
    __syncthreads();
}

// the sum of target number t of the block: the streams' in order
template <int kI, int kW>
__device__ __forceinline__ float3 direct_target_sum(DirectShared<kI, kW> &sh, int t) {
    float3 a = make_float3(0.0f, 0.0f, 0.0f);
    for (int w = 0; w < kDirectStreams; ++w) {
        const float *at = sh.sums() + w * (3 * 32 * kI) + t;
        a.x += at[0];
        a.y += at[32 * kI];
        a.z += at[64 * kI];
    }
    return a;
}

}  // namespace nbgb
