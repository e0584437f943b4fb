// k_collide.cu -- the collision update of a single system
// (update_collision_local, kernels/collision_update.cl:17-83;
// collide_device.cuh).  It reads the positions the integrator of the same step
// wrote, as the reference runs it after the force kernel
// (src/MyApp.cpp:593-596).  A step that failed keeps its step-start state, so
// the update does not run then.
//
// Three forms, all giving the same bits:
//   warp   one target per warp, 32 bodies tested at a time, all n bodies;
//   block  one target per thread, all n bodies in staged tiles;
//   grid   a target meets only the bodies of the 27 grid cells around it.
// The pair tests of the first two are all there is to their time (n^2); the
// grid leaves about 27 h^3 n / V candidates a target and is bound by its
// scattered reads of them and, below 100,000 bodies, by its six launches.
// Unit ball, tree systems, GB300, warp or block form against grid: N = 20,000 0.49
// -> 0.043 ms, 60,001 3.38 -> 0.063, 131,072 8.54 -> 0.117.  What the grid cannot
// serve takes as long as without it (k_grid_rest_few, k_grid_rest).
#include <algorithm>

#include "collide_device.cuh"
#include "launch.cuh"

namespace nbgb {

__global__ void __launch_bounds__(kCollideWarps * 32) k_collision_warp(DevSim s) {
    wait_for_previous();
    if (read_status(s.ctrl)) return;  // warp-uniform
    const int lane = threadIdx.x & 31;
    collide_warp(s.body_next, s.vel, s.n, blockIdx.x * kCollideWarps + (threadIdx.x >> 5), lane);
}

// ---------------------------------------------------------------------------
// Grid form.  Cells of edge h = 17/16 of the contact distance: the index of a
// body along an axis is floor(x / h), formed in FP32.  Two bodies in contact
// are at most 16/17 (1 + 2^-22) cells apart along each axis, and the rounding
// of x / h moves each by at most 2^-24 |x / h| < 1/64 for |x / h| < 2^18, so
// their indices differ by at most one.  A system with a body beyond that, or
// one that is not finite (its distance is NaN, which the reference counts as
// a contact with everything), takes the block form.
//
// The cells live in a hash table of 2^k >= n buckets; cells that follow one
// another along x have buckets that follow one another, so a row of three
// cells is usually one range.  A candidate counts only in the row of its true
// cell, so cells that share a bucket give no body twice.
//
// A target lists its contacts (at most kGridContacts), then applies them in
// ascending body index, as the reference's loop does.  Targets with more
// contacts go to an overflow list that the last kernel serves by the other two
// forms.
// ---------------------------------------------------------------------------
constexpr int kGridThreads = 128;
constexpr int kGridContacts = 64;
// A target with too many bodies around it goes to the overflow list at once: a
// thread takes 0.4 us a candidate where nothing hides its latencies, the warp form
// about n^2 / 2^20 us for all n targets, of which the candidates may take two fifths;
// and with 16 kGridContacts around it, it has more contacts than its list holds.
// Targets ask for it where some bucket holds more than its share of that, and more
// than kGridQuiet.
__device__ __forceinline__ int grid_crowd(int n) { return (int)min((long long)n * n >> 20, 16LL * kGridContacts); }
constexpr int kGridQuiet = 8;
constexpr int kScanBuckets = 1024;  // buckets per block of the scan: consecutive in memory
constexpr float kGridLimit = 262144.0f;

__device__ __forceinline__ float grid_inv() { return __fdiv_rn(16.0f, __fmul_rn(17.0f, contact_distance())); }

struct GridCell {
    int x, y, z;
};
// false when the body has no cell: not finite, or too far out
__device__ __forceinline__ bool grid_cell(const float4 p, float inv, GridCell &c) {
    const float x = p.x * inv, y = p.y * inv, z = p.z * inv;
    if (!(fabsf(x) < kGridLimit && fabsf(y) < kGridLimit && fabsf(z) < kGridLimit)) return false;
    c = GridCell{__float2int_rd(x), __float2int_rd(y), __float2int_rd(z)};
    return true;
}
__device__ __forceinline__ unsigned grid_row(int y, int z) {
    unsigned h = (unsigned)y * 0x9E3779B1u ^ (unsigned)z * 0x85EBCA77u;
    h ^= h >> 15;
    return h * 0x2C1B3C6Du;
}

__global__ void k_grid_count(DevSim s, CollideGrid g) {
    if (read_status(s.ctrl)) return;
    const float inv = grid_inv();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < s.n; i += gridDim.x * blockDim.x) {
        GridCell c;
        if (!grid_cell(s.body_next[i], inv, c)) {
            g.ctl[kGridNoCell] = 1;
            continue;
        }
        g.rank[i] = atomicAdd(&g.count[(grid_row(c.y, c.z) + (unsigned)c.x) & g.mask], 1);
    }
}

// start of every bucket: a block lays its kScanBuckets buckets end to end at a
// place from one atomic
__global__ void __launch_bounds__(kScanBuckets / 4) k_grid_scan(DevSim s, CollideGrid g) {
    wait_for_previous();
    if (read_status(s.ctrl)) return;  // grid-uniform, before any barrier
    __shared__ int warp_tot[kScanBuckets / 128];
    __shared__ int base;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int at = blockIdx.x * (kScanBuckets / 4) + threadIdx.x;
    const int4 c = reinterpret_cast<const int4 *>(g.count)[at];
    const int sum = c.x + c.y + c.z + c.w;
    if (max(max(c.x, c.y), max(c.z, c.w)) > max(kGridQuiet, grid_crowd(s.n) / 27)) g.ctl[kGridCrowded] = 1;
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int k = 0; k < kScanBuckets / 128; ++k) {
            const int v = warp_tot[k];
            warp_tot[k] = t;
            t += v;
        }
        base = atomicAdd(&g.ctl[kGridCursor], t);
    }
    __syncthreads();
    const int b = base + warp_tot[w] + incl - sum;
    reinterpret_cast<int4 *>(g.start)[at] = make_int4(b, b + c.x, b + c.x + c.y, b + c.x + c.y + c.z);
}

// bodies into their buckets: {x, y, z, index}
__global__ void k_grid_place(DevSim s, CollideGrid g) {
    wait_for_previous();
    if (read_status(s.ctrl) || g.ctl[kGridNoCell]) return;
    const float inv = grid_inv();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < s.n; i += gridDim.x * blockDim.x) {
        const float4 p = s.body_next[i];
        GridCell c;
        grid_cell(p, inv, c);
        g.body[g.start[(grid_row(c.y, c.z) + (unsigned)c.x) & g.mask] + g.rank[i]] =
            make_float4(p.x, p.y, p.z, __int_as_float(i));
    }
}

// one target per thread, targets in bucket order (neighbours read the same
// candidates)
__global__ void __launch_bounds__(kGridThreads) k_grid_collide(DevSim s, CollideGrid g) {
    wait_for_previous();
    __shared__ int found[kGridContacts][kGridThreads];
    if (read_status(s.ctrl) || g.ctl[kGridNoCell]) return;
    const int t = blockIdx.x * kGridThreads + threadIdx.x;
    if (t >= s.n) return;
    const float4 me = g.body[t];
    const int i = __float_as_int(me.w);
    const float inv = grid_inv(), rr = contact_distance();
    GridCell c;
    grid_cell(me, inv, c);
    // the rows' three buckets: one range when the scan laid them end to end
    int cnt = 0, crowd = 8 * kGridContacts;  // about that many bodies are around a target with kGridContacts contacts
    if (g.ctl[kGridCrowded]) {
        crowd = 0;
#pragma unroll
        for (int row = 0; row < 9; ++row) {
            const unsigned b0 = (grid_row(c.y + row / 3 - 1, c.z + row % 3 - 1) + (unsigned)(c.x - 1)) & g.mask;
            if ((b0 & (kScanBuckets - 1)) + 2 < kScanBuckets) crowd += g.start[b0 + 2] + g.count[b0 + 2] - g.start[b0];
        }
        if (crowd > grid_crowd(s.n)) cnt = kGridContacts + 1;
    }
    for (int row = 0; row < 9 && cnt <= kGridContacts; ++row) {
        const int cy = c.y + row / 3 - 1, cz = c.z + row % 3 - 1;
        const unsigned b0 = (grid_row(cy, cz) + (unsigned)(c.x - 1)) & g.mask;
        const bool whole = (b0 & (kScanBuckets - 1)) + 2 < kScanBuckets;
        for (int part = 0; part < (whole ? 1 : 3); ++part) {
            const unsigned first = (b0 + part) & g.mask, last = whole ? b0 + 2 : first;
            const int end = g.start[last] + g.count[last];
            for (int k = g.start[first]; k < end && cnt <= kGridContacts; ++k) {
                const float4 q = g.body[k];
                const int j = __float_as_int(q.w);
                if (j == i || !in_contact(me, q, rr, true)) continue;
                GridCell d;
                grid_cell(q, inv, d);
                if (d.y != cy || d.z != cz || abs(d.x - c.x) > 1 || (!whole && d.x != c.x - 1 + part)) continue;
                if (cnt < kGridContacts) found[cnt][threadIdx.x] = j;
                ++cnt;
            }
        }
    }
    if (cnt == 0) return;
    if (cnt > kGridContacts) {
        g.rank[atomicAdd(&g.ctl[kGridOverflow], 1)] = i;  // the ranks are no longer needed
        atomicAdd(reinterpret_cast<unsigned long long *>(&g.ctl[kGridAround]), (unsigned long long)crowd);
        return;
    }
    float4 v = s.vel[i];
    for (int k = 0; k < cnt; ++k) {  // ascending body index
        int best = k, low = found[k][threadIdx.x];
        for (int m = k + 1; m < cnt; ++m) {
            const int j = found[m][threadIdx.x];
            if (j < low) {
                low = j;
                best = m;
            }
        }
        found[best][threadIdx.x] = found[k][threadIdx.x];
        reflect(me, s.body_next[low], v);
    }
    s.vel[i] = v;
}

// What the grid left: every target when some body has no cell, else the targets
// of the overflow list.  Few of them take one warp each, many one thread each, as
// collide_warp_form_below decides between whole systems.
//
// The warps' form.  Targets' times differ with their contacts, so after the first
// one a warp draws the next; a block per eight targets did as well, but blocks that
// find nothing to do cost 6 us at 38,000 bodies.  Not inlined: around the loop the
// compiler gives it 42 registers, or spills (38,000 targets, one body far out: 1.57
// ms, with 42 registers 1.89, a warp a target and no grid before it 1.47).
__device__ __noinline__ void collide_one(const float4 *pos, float4 *vel, int n, int i) {
    collide_warp(pos, vel, n, i, threadIdx.x & 31);
}
__device__ __forceinline__ void rest_by_warps(const DevSim &s, const CollideGrid &g, bool all, int cnt) {
    const int warps = gridDim.x * kCollideWarps;
    for (int k = blockIdx.x * kCollideWarps + (threadIdx.x >> 5); k < cnt;) {
        collide_one(s.body_next, s.vel, s.n, all ? k : g.rank[k]);
        if (cnt <= warps) return;
        if ((threadIdx.x & 31) == 0) k = warps + atomicAdd(&g.ctl[kGridNext], 1);
        k = __shfl_sync(0xffffffffu, k, 0);
    }
}
// systems that cannot have many
__global__ void __launch_bounds__(kCollideWarps * 32, 8) k_grid_rest_few(DevSim s, CollideGrid g) {
    wait_for_previous();
    if (read_status(s.ctrl)) return;  // warp-uniform
    const bool all = g.ctl[kGridNoCell] != 0;
    rest_by_warps(s, g, all, all ? s.n : g.ctl[kGridOverflow]);
}
// Systems that may have many.  A target that meets few bodies is the warps' (32 of
// its pairs a step), one that meets thousands a thread's: its reflections follow one
// another, and 32 targets share a warp.  An eighth of the bodies around a target
// (`around`, all targets together) are its contacts.  In us, from the times of both
// forms alone: a warp's step 0.1, its contact 0.15, up to 24 warps per SM; a body of
// the blocks' tiles 0.05, up to three blocks per SM, their contact 0.3.  (60,001
// bodies, an eighth in a core: warps 2.6 ms, blocks 3.9; 59,157 bodies of a cusp 92
// and 11.)
__device__ __forceinline__ bool warps_are_faster(int n, int cnt, unsigned long long around, int sm_count) {
    const int warps = min(min(cnt, (int)gridDim.x * kCollideWarps), 24 * sm_count);
    const float contacts = 0.125f * (float)around, targets = (float)cnt;
    return (0.1f * targets * (float)n / 32.0f + 0.15f * contacts) / (float)warps <
           0.05f * (float)n * fmaxf(1.0f, targets / (float)(3 * kCollideThreads * sm_count)) + 0.3f * contacts / targets;
}
__global__ void __launch_bounds__(kCollideThreads, 8) k_grid_rest(DevSim s, CollideGrid g, const int *order,
                                                                  int sm_count) {
    wait_for_previous();
    if (read_status(s.ctrl)) return;  // block-uniform, before any barrier
    const bool all = g.ctl[kGridNoCell] != 0;
    const int cnt = all ? s.n : g.ctl[kGridOverflow];
    if (cnt == 0) return;
    if (!all && warps_are_faster(s.n, cnt, *reinterpret_cast<const unsigned long long *>(&g.ctl[kGridAround]), sm_count))
        return rest_by_warps(s, g, all, cnt);
    if ((int)blockIdx.x * kCollideThreads >= cnt) return;
    collide_block(s.body_next, s.vel, all ? order : g.rank, cnt, s.n, blockIdx.x * kCollideThreads, s.ctrl);
}

cudaError_t launch_collision(const DevSim &s, const CollideGrid &g, int tree, int sm_count, cudaStream_t st,
                             int *launches) {
    if (!g.count) {
        *launches = 1;
        const int blocks = (s.n + kCollideWarps - 1) / kCollideWarps;
        // early (3 us) only where no two blocks need share an SM: behind the direct sums
        // early blocks are placed unevenly (launch.cuh; direct systems of 2,859 bodies
        // all in contact 0.64 ms, early 0.99; spread out 38 us, early 36)
        if (blocks <= sm_count) return launch_next(k_collision_warp, blocks, kCollideWarps * 32, st, s);
        k_collision_warp<<<blocks, kCollideWarps * 32, 0, st>>>(s);
        return cudaGetLastError();
    }
    *launches = 5;
    // counts and the control words, one array
    cudaError_t e = cudaMemsetAsync(g.count, 0, sizeof(int) * ((size_t)g.mask + 1 + kGridCtl), st);
    if (e != cudaSuccess) return e;
    const int blocks = std::min((s.n + 255) / 256, sm_count * 8);
    k_grid_count<<<blocks, 256, 0, st>>>(s, g);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = launch_next(k_grid_scan, (int)((g.mask + 1) / kScanBuckets), kScanBuckets / 4, st, s, g);
    if (e == cudaSuccess) e = launch_next(k_grid_place, blocks, 256, st, s, g);
    if (e == cudaSuccess)
        e = launch_next(k_grid_collide, (s.n + kGridThreads - 1) / kGridThreads, kGridThreads, st, s, g);
    if (e != cudaSuccess) return e;
    const int few = collide_warp_form_below(sm_count) * kCollideThreads;
    if (s.n < few)
        return launch_next(k_grid_rest_few, std::min((s.n + kCollideWarps - 1) / kCollideWarps, 8 * sm_count),
                           kCollideWarps * 32, st, s, g);
    // not early, so that the block form's few long blocks spread evenly (launch.cuh;
    // 60,001 bodies, one far out: 3.50 ms, early 4.02)
    k_grid_rest<<<(s.n + kCollideThreads - 1) / kCollideThreads, kCollideThreads, 0, st>>>(
        s, g, tree ? s.sorted : nullptr, sm_count);
    return cudaGetLastError();
}

}  // namespace nbgb
