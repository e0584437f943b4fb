// k_build.cu -- bounding box, octree, centres of mass and in-order sort of a
// single system with the cubic-root tree, from sorted octant paths.
//
// Reference stages: boundary_reduce, init, build_tree, saturate_tree and the
// empty sort (kernels/*.cl).  The octree is a function of the points: a cell
// exists exactly where two bodies share its octant path.  So the bodies are
// sorted by path -- which is the in-order sort the walk needs -- and every cell
// follows from two neighbours' common levels; no thread waits for another, and
// the sums of a cell are formed where its bodies already lie in shared memory.
// The tree, its sums (children in slot order, each operation rounded as in
// summarize_from) and the sort are those of the insertions, bit for bit; only
// the cells' numbering differs.
//
//   k_box     bounding box; resets the step's counters
//   k_path    octant path of every body, 3 bits a level, 21 levels; above
//             kRankAll bodies also its region (the first `levels` levels) and
//             its place there
//   k_scan    start of every region
//   k_place   bodies into their regions
//   k_rank    place of every body among those of its region (or, without
//             regions, among all)
//   k_cells   cells that start at each body, their numbers
//   k_link    tiles of kTile sorted bodies: the cells that lie inside one tile
//             bottom up, and the links of the few that do not
//   k_top     those few, by arrival counters
//
// Bodies that 21 levels do not part, regions too crowded to rank (bodies far
// out in a wide box) and the wait-cap test hook take the insertions instead
// (bh_device.cuh), all inside k_top's launch: the earlier kernels set
// ctrl->insert and the later ones leave at once.
//
// What bounds it: launches and chains of dependent L2 accesses up to some
// 100,000 bodies (4 to 9 us a kernel, 25 in k_top, whose longest chain has a
// cell per level), beyond that k_link's block barriers between levels (issue
// slots half used) and the scattered writes of k_place.  Insertions from five
// prepared top levels, the summarisation by arrival counters and the sort by
// waits took, against this (GB300, us): 6,007 bodies 107 -> 66; 100,003 with
// quadrupoles 215 -> 98; 262,144 196 -> 114; 4,194,304 with quadrupoles 1,718 ->
// 1,080.
#include <algorithm>

#include "bh_device.cuh"
#include "launch.cuh"

namespace nbgb {

typedef unsigned long long u64;
constexpr int kPathLevels = 21;
constexpr int kTile = 256;          // sorted bodies per block of k_cells and k_link, one per thread
constexpr int kScanThreads = 1024;  // k_scan: eight regions per thread
constexpr int kScanRegions = 8 * kScanThreads;

// ---------------------------------------------------------------------------
// bbox: exact component-wise min/max as order-preserving integer keys.  The
// reference's reduction samples only 2*WG bodies as wired (src/MyApp.cpp:282).
// The block that finishes last reduces the blocks' results and sets what a
// step starts from (init, kernels/init.cl:26-33: the root; the counters).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_box(DevSim s, BuildScratch b) {
    __shared__ unsigned red[8][6];
    __shared__ int last;
    Ctrl *c = s.ctrl;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned v[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
    auto block_reduce = [&]() {
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            v[k] = k < 3 ? __reduce_min_sync(0xffffffffu, v[k]) : __reduce_max_sync(0xffffffffu, v[k]);
            if (lane == 0) red[w][k] = v[k];
        }
        __syncthreads();
        unsigned r = 0;
        if (threadIdx.x < 6) {
            const int k = threadIdx.x;
            r = red[0][k];
            for (int j = 1; j < 8; ++j) r = k < 3 ? min(r, red[j][k]) : max(r, red[j][k]);
        }
        return r;
    };
    int bad = -1;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < s.n; i += gridDim.x * blockDim.x) {
        const float4 p = __ldg(&s.body_cur[i]);
        if (!(isfinite(p.x) && isfinite(p.y) && isfinite(p.z))) bad = i;
        const unsigned kx = f2key(p.x), ky = f2key(p.y), kz = f2key(p.z);
        v[0] = min(v[0], kx);
        v[1] = min(v[1], ky);
        v[2] = min(v[2], kz);
        v[3] = max(v[3], kx);
        v[4] = max(v[4], ky);
        v[5] = max(v[5], kz);
    }
    if (bad >= 0) set_status(c, kStNonFinite, bad);
    const unsigned r = block_reduce();
    if (threadIdx.x < 6) {
        b.box[blockIdx.x * 6 + threadIdx.x] = r;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&b.ctl[kBuildBoxes], 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] = k < 3 ? 0xFFFFFFFFu : 0u;
    for (int j = threadIdx.x; j < (int)gridDim.x; j += blockDim.x)
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const unsigned x = __ldcg(&b.box[j * 6 + k]);
            v[k] = k < 3 ? min(v[k], x) : max(v[k], x);
        }
    const unsigned all = block_reduce();
    if (threadIdx.x < 6) c->bbox_key[threadIdx.x] = all;
    b.total[threadIdx.x] = 0;  // kScanBlocks = blockDim.x
    if (threadIdx.x < 8) s.child[s.cap * 8 + threadIdx.x] = kEmpty;
    if (threadIdx.x == 0) {
        c->bottom = s.n + s.cap;
        c->max_depth = 0;
        c->work = 0;
        c->insert = c->spin_cap > 0;  // the hook caps the insertions' waits
        s.arrive[s.cap] = 0;
        s.start[s.cap] = 0;
        s.count[s.cap] = 0;
        s.parent[s.cap] = -1;
        b.ctl[kBuildBoxes] = 0;
        b.ctl[kBuildBarrier] = 0;
        b.ctl[kBuildTop] = 1;
        b.top[0] = s.n + s.cap;
        *reinterpret_cast<u64 *>(&b.ctl[kBuildPairs]) = 0;
    }
}

// ---------------------------------------------------------------------------
// paths
// ---------------------------------------------------------------------------
__device__ __forceinline__ u64 octant_path(GeoCube g, const float4 P) {
    u64 key = 0;
#pragma unroll
    for (int l = 0; l < kPathLevels; ++l) {
        key = key * 8 + (u64)g.octant(P.x, P.y, P.z);
        g.descend(P.x, P.y, P.z);
    }
    return key;
}
__device__ __forceinline__ int region_of(u64 key, int levels) { return (int)(key >> (3 * (kPathLevels - levels))); }
// levels two paths share: the level of the deepest cell that holds both
__device__ __forceinline__ int common_levels(u64 a, u64 b) {
    const u64 x = a ^ b;
    return x ? (__clzll((long long)x) - 1) / 3 : kPathLevels;
}
__device__ __forceinline__ int octant_at(u64 key, int level) { return (int)(key >> (3 * (kPathLevels - 1 - level))) & 7; }
__device__ __forceinline__ bool build_off(const Ctrl *c) { return read_status(c) != 0 || c->insert != 0; }

__global__ void __launch_bounds__(256) k_path(DevSim s, BuildScratch b) {
    wait_for_previous();
    if (build_off(s.ctrl)) return;
    float box[6];
    load_box(s.ctrl, box);
    const GeoCube root = GeoCube::root(box);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < s.n; i += gridDim.x * blockDim.x) {
        const u64 key = octant_path(root, __ldg(&s.body_cur[i]));
        b.path[i] = key;
        if (b.levels) b.rank[i] = atomicAdd(&b.count[region_of(key, b.levels)], 1);
    }
}

// Exclusive scan of the region counts (a block adds up the totals of the
// blocks before it as they appear; all blocks of the grid, at most kScanBlocks,
// are resident together, and take as many chunks of kScanRegions as that
// needs).  Clears the counts for the next step and adds up the pairs that
// ranking the regions will compare.
inline __host__ __device__ int scan_chunks(int levels) {
    const int chunks = ((1 << (3 * levels)) + kScanRegions - 1) / kScanRegions;
    return (chunks + kScanBlocks - 1) / kScanBlocks;
}
__global__ void __launch_bounds__(kScanThreads, 2) k_scan(DevSim s, BuildScratch b) {
    wait_for_previous();
    __shared__ int warp_tot[32];
    __shared__ u64 warp_sq[32];
    __shared__ int before;
    if (__syncthreads_or(build_off(s.ctrl))) return;  // a wait that gave up elsewhere stops whole blocks
    const int regions = 1 << (3 * b.levels), chunks = scan_chunks(b.levels);
    const int begin = blockIdx.x * chunks * kScanRegions;
    int4 c0, c1;
    auto load = [&](int chunk) {
        const int at = begin + chunk * kScanRegions + threadIdx.x * 8;
        c0 = c1 = make_int4(0, 0, 0, 0);
        if (at < regions) {
            c0 = reinterpret_cast<const int4 *>(&b.count[at])[0];
            c1 = reinterpret_cast<const int4 *>(&b.count[at])[1];
        }
        return c0.x + c0.y + c0.z + c0.w + c1.x + c1.y + c1.z + c1.w;
    };
    u64 sq = 0;
    int sum = 0;
    for (int chunk = 0; chunk < chunks; ++chunk) {
        sum += load(chunk);
        sq += (u64)c0.x * c0.x + (u64)c0.y * c0.y + (u64)c0.z * c0.z + (u64)c0.w * c0.w + (u64)c1.x * c1.x +
              (u64)c1.y * c1.y + (u64)c1.z * c1.z + (u64)c1.w * c1.w;
    }
    int total;
    int ex = block_exclusive_sum(sum, warp_tot, &total);
    if (threadIdx.x == 0) st_volatile(&b.total[blockIdx.x], total + 1);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0) warp_sq[threadIdx.x >> 5] = sq;
    __syncthreads();
    if (threadIdx.x >= 32 && threadIdx.x < 64) {
        sq = warp_sq[threadIdx.x & 31];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (threadIdx.x == 32) atomicAdd(reinterpret_cast<u64 *>(&b.ctl[kBuildPairs]), sq);
    }
    if (threadIdx.x < 32) {
        int acc = 0;
        for (int k = threadIdx.x; k < (int)blockIdx.x; k += 32) {
            int t = ld_volatile(&b.total[k]);
            for (long long spins = 0; t == 0; t = ld_volatile(&b.total[k]))
                if (++spins > kSpinCap) {
                    set_status(s.ctrl, kStSpinTimeout, k);
                    break;
                }
            acc += t - 1;
        }
        acc = __reduce_add_sync(0xffffffffu, acc);
        if (threadIdx.x == 0) before = acc;
    }
    __syncthreads();
    int base = before;
    for (int chunk = 0; chunk < chunks; ++chunk) {
        if (chunks > 1) ex = block_exclusive_sum(load(chunk), warp_tot, &total);  // one chunk: still in registers
        const int at = begin + chunk * kScanRegions + threadIdx.x * 8;
        if (at < regions) {
            int4 o0, o1;
            o0.x = base + ex;
            o0.y = o0.x + c0.x;
            o0.z = o0.y + c0.y;
            o0.w = o0.z + c0.z;
            o1.x = o0.w + c0.w;
            o1.y = o1.x + c1.x;
            o1.z = o1.y + c1.y;
            o1.w = o1.z + c1.z;
            int4 *p = reinterpret_cast<int4 *>(&b.start[at]);
            p[0] = o0;
            p[1] = o1;
            p = reinterpret_cast<int4 *>(&b.count[at]);
            p[0] = p[1] = make_int4(0, 0, 0, 0);
        }
        base += total;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) b.start[regions] = s.n;
}

// more pairs than this a body and the insertions are faster
constexpr int kPairsPerBody = 512;
__device__ __forceinline__ bool too_crowded(const DevSim &s, const BuildScratch &b) {
    return *reinterpret_cast<const volatile u64 *>(&b.ctl[kBuildPairs]) > (u64)s.n * kPairsPerBody;
}

__global__ void __launch_bounds__(256) k_place(DevSim s, BuildScratch b) {
    wait_for_previous();
    if (build_off(s.ctrl) || too_crowded(s, b)) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < s.n; i += gridDim.x * blockDim.x) {
        const u64 key = b.path[i];
        const int at = b.start[region_of(key, b.levels)] + b.rank[i];
        b.placed[at] = key;
        b.who[at] = i;
    }
}

// Place of every body among those of its region: the number of smaller paths
// there, equal ones in the order they lie.  A block's regions lie end to end and
// pass through shared memory.  Equal paths (21 levels do not part the bodies)
// end up side by side, where k_cells sees them.
constexpr int kRankChunk = 1024;
__global__ void __launch_bounds__(256) k_rank(DevSim s, BuildScratch b) {
    wait_for_previous();
    __shared__ u64 sh[kRankChunk];
    if (__syncthreads_or(build_off(s.ctrl))) return;  // other blocks of this kernel may set `insert`
    if (too_crowded(s, b)) {                          // grid-uniform
        s.ctrl->insert = 1;
        return;
    }
    const int first = blockIdx.x * blockDim.x, last = min(s.n, first + (int)blockDim.x) - 1;
    const int i = first + threadIdx.x;
    const u64 key = b.placed[min(i, last)];
    const int r = region_of(key, b.levels);
    const int lo = b.start[r], hi = i < s.n ? b.start[r + 1] : lo;
    const int block_lo = b.start[region_of(b.placed[first], b.levels)];
    const int block_hi = b.start[region_of(b.placed[last], b.levels) + 1];
    int less = 0;
    for (int at = block_lo; at < block_hi; at += kRankChunk) {
        __syncthreads();
        for (int j = threadIdx.x; j < min(kRankChunk, block_hi - at); j += blockDim.x) sh[j] = b.placed[at + j];
        __syncthreads();
        const int j0 = max(lo - at, 0), j1 = min(hi - at, kRankChunk), own = i - at;
#pragma unroll 4
        for (int j = j0; j < min(j1, own); ++j) less += sh[j] <= key;
#pragma unroll 4
        for (int j = max(j0, own + 1); j < j1; ++j) less += sh[j] < key;
    }
    if (i >= s.n) return;
    s.sorted[lo + less] = b.who[i];
    b.path[lo + less] = key;
}

// Small systems: 32 bodies a block against all n, an eighth per warp.
constexpr int kRankWarps = 8;
constexpr int kRankPart = 512;  // loads in flight together; n <= kRankAll takes two parts
__global__ void __launch_bounds__(32 * kRankWarps) k_rank_all(DevSim s, BuildScratch b) {
    wait_for_previous();
    __shared__ u64 sh[kRankWarps][kRankPart];
    __shared__ int part[kRankWarps][32];
    if (build_off(s.ctrl)) return;  // grid-uniform: only earlier kernels set either
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, n = s.n;
    const int first = blockIdx.x * 32, i = first + lane;
    const u64 key = i < n ? b.path[i] : 0;
    const int per = (n + kRankWarps - 1) / kRankWarps, lo = w * per, hi = min(n, lo + per);
    int less = 0;
    for (int at = lo; at < hi; at += kRankPart) {
        const int m = min(kRankPart, hi - at), m16 = (m + 15) & ~15;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < kRankPart / 32; ++k)  // beyond the part: larger than every path
            sh[w][32 * k + lane] = 32 * k + lane < m ? b.path[at + 32 * k + lane] : ~0ull;
        __syncwarp();
        if (at + m <= first) {
            // every path here comes before the block's bodies: equal ones count
#pragma unroll 16
            for (int j = 0; j < m16; ++j) less += sh[w][j] <= key;
        } else if (at >= first + 32) {
#pragma unroll 16
            for (int j = 0; j < m16; ++j) less += sh[w][j] < key;
        } else {
            for (int j = 0; j < m; ++j) less += at + j < i ? sh[w][j] <= key : sh[w][j] < key;
        }
    }
    part[w][lane] = less;
    __syncthreads();
    if (w > 0 || i >= n) return;
    less = 0;
#pragma unroll
    for (int k = 0; k < kRankWarps; ++k) less += part[k][lane];
    s.sorted[less] = i;
    b.placed[less] = key;
}

// ---------------------------------------------------------------------------
// Cells.  With d(i) = the levels bodies i and i+1 share, d(-1) = d(n-1) = -1, the
// cells whose first body is i are those of the levels max(d(i-1), 0) + 1 .. d(i):
// numbered downwards from base[i].  (The root is level 0 and always there.)
// A cell of level l that starts at i ends at the first e >= i with d(e) < l; the
// places with d = l inside it part its children.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int cell_number(int base, int lo, int level) { return base - (level - lo - 1); }

// first of keys[0, m) (ascending) that shares `level` levels with `key`, which
// the last one does
template <class Key>
__device__ __forceinline__ int first_sharing(Key keys, int m, u64 key, int level) {
    const int sh = 3 * (kPathLevels - level);
    int lo = 0, hi = m - 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if ((keys(mid) >> sh) < (key >> sh)) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Four tiles a block, four bodies a thread: the block's chain of waits (paths,
// scan, the numbers' atomic) is what it takes, so a block does more.
constexpr int kCellTiles = 4;
constexpr int kCellBodies = kCellTiles * kTile;
__global__ void __launch_bounds__(kTile) k_cells(DevSim s, BuildScratch b, const u64 *__restrict__ path) {
    wait_for_previous();
    __shared__ u64 key_sh[kCellBodies + 2];  // the paths of bodies a - 1 .. a + kCellBodies
    __shared__ int base_sh[kCellBodies];
    __shared__ int warp_tot[32];
    __shared__ int first, deepest;
    if (__syncthreads_or(build_off(s.ctrl))) return;  // an overflow elsewhere stops whole blocks
    Ctrl *c = s.ctrl;
    const int t = threadIdx.x, n = s.n, a = blockIdx.x * kCellBodies, m = min(kCellBodies, n - a);
    if (t == 0) deepest = 0;
    for (int k = t; k < m + 2; k += kTile) {
        const int i = a - 1 + k;
        if (i >= 0 && i < n) key_sh[k] = path[i];
    }
    __syncthreads();
    // levels that local bodies k - 1 and k share
    auto shared_levels = [&](int k) {
        return a + k > 0 && a + k < n ? common_levels(key_sh[k], key_sh[k + 1]) : -1;
    };
    int d[5], lo[4], mine[4], sum = 0, deep = -1;
#pragma unroll
    for (int k = 0; k < 5; ++k) d[k] = 4 * t + k <= m ? shared_levels(4 * t + k) : -1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        lo[k] = max(d[k], 0);
        mine[k] = 4 * t + k < m ? max(0, d[k + 1] - lo[k]) : 0;
        sum += mine[k];
        deep = max(deep, d[k + 1]);
    }
    if (deep >= kPathLevels) c->insert = 1;  // equal paths: the later kernels leave the build to the insertions
    int total;
    int ex = block_exclusive_sum(sum, warp_tot, &total);
    deep = __reduce_max_sync(0xffffffffu, deep);
    if ((t & 31) == 0 && deep > 0) atomicMax(&deepest, deep);
    if (t == 0) first = atomicSub(&c->bottom, total);
    __syncthreads();
    if (t == 0 && deepest > 0) atomicMax(&c->max_depth, deepest);
    if (first - total < n) {  // block-uniform: more cells than the capacity
        if (t == 0) set_status(c, kStCellOverflow, a);
        return;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (4 * t + k < m) {
            base_sh[4 * t + k] = first - 1 - ex;
            b.base[a + 4 * t + k] = first - 1 - ex;
        }
        ex += mine[k];
    }
    __syncthreads();
    // the cells that start in a tile and go on beyond it: ancestors of its last
    // body, one tile per warp, one level per lane
    const int w = t >> 5, level = t & 31, t0 = w * kTile;
    if (w < kCellTiles && t0 < m) {
        const int t1 = min(t0 + kTile, m);  // the tile's local bodies
        const int end = shared_levels(t1);
        if (level >= 1 && level <= end && end < kPathLevels) {
            const int st =
                t0 + first_sharing([&](int k) { return key_sh[t0 + 1 + k]; }, t1 - t0, key_sh[t1], level);
            const int pre = shared_levels(st);
            if (pre < level) {
                const int cell = cell_number(base_sh[st], max(pre, 0), level), k = cell - n;
                int4 *row = reinterpret_cast<int4 *>(&s.child[k * 8]);
                row[0] = row[1] = make_int4(kEmpty, kEmpty, kEmpty, kEmpty);
                s.arrive[k] = 0;
                s.start[k] = 1;  // completed by k_top
                b.top[atomicAdd(&b.ctl[kBuildTop], 1)] = cell;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// k_link.  An item of the tile is a body or a completed cell at its first body's
// place; the levels run from the deepest to 1, and a cell that ends inside the
// tile takes its items together (summation as in summarize_from) and becomes
// one.  What is left belongs to cells that reach beyond the tile: each item is
// entered in its parent's row, and so is each such cell that starts here.
// ---------------------------------------------------------------------------
// A cell is summed by eight lanes, one per child: the children's data and the
// rows they are stored in move a whole line at a time, and the sums go through
// the lanes in slot order.
struct CellSums {
    float M, X, Y, Z;  // mass and centre
    int cnt;
};
// group: the mask of the eight lanes; mask: which of the
// eight hold a child (in slot order)
__device__ __forceinline__ CellSums sum_children(unsigned group, unsigned mask, const float4 p, int cnt) {
    const float wx = __fmul_rn(p.x, p.w), wy = __fmul_rn(p.y, p.w), wz = __fmul_rn(p.z, p.w);
    float M = 0.0f, cx = 0.0f, cy = 0.0f, cz = 0.0f;
    int total = 0;
    for (int q = 0; mask >> q; ++q) {
        const float vm = __shfl_sync(group, p.w, q, 8), vx = __shfl_sync(group, wx, q, 8),
                    vy = __shfl_sync(group, wy, q, 8), vz = __shfl_sync(group, wz, q, 8);
        const int vc = __shfl_sync(group, cnt, q, 8);
        if ((mask >> q) & 1u) {
            M = __fadd_rn(M, vm);
            cx = __fadd_rn(cx, vx);
            cy = __fadd_rn(cy, vy);
            cz = __fadd_rn(cz, vz);
            total += vc;
        }
    }
    const float inv = __frcp_rn(M);
    return CellSums{M, __fmul_rn(cx, inv), __fmul_rn(cy, inv), __fmul_rn(cz, inv), total};
}
// the quadrupole sums about the centre; q[k] of lane j: its child's moments in,
// the cell's out
__device__ __forceinline__ void sum_quadrupoles(unsigned group, unsigned mask, const float4 p, const CellSums &c,
                                                float (&q)[6]) {
    float e0 = 0.0f, e1 = 0.0f, e2 = 0.0f, e3 = 0.0f, e4 = 0.0f, e5 = 0.0f;
    quadrupole_term(p, c.X, c.Y, c.Z, make_float4(q[0], q[1], q[2], q[3]), q[4], q[5], e0, e1, e2, e3, e4, e5);
    const float e[6] = {e0, e1, e2, e3, e4, e5};
#pragma unroll
    for (int k = 0; k < 6; ++k) q[k] = 0.0f;
    for (int m = 0; mask >> m; ++m) {
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const float x = __shfl_sync(group, e[k], m, 8);
            if ((mask >> m) & 1u) q[k] = __fadd_rn(q[k], x);
        }
    }
}

template <bool kQuad>
__global__ void __launch_bounds__(kTile) k_link(DevSim s, BuildScratch b, const u64 *__restrict__ path) {
    wait_for_previous();
    __shared__ float4 pm[kTile];
    __shared__ float q6[kQuad ? 6 : 1][kQuad ? kTile : 1];
    __shared__ u64 key_sh[kTile];
    __shared__ int base_sh[kTile], node[kTile], cnt_sh[kTile];
    __shared__ int item[kTile];  // of the item that starts here: (d(its end) + 1) << 16 | its end
    __shared__ short list[kTile];
    __shared__ signed char d[kTile + 1];  // d[t + 1] = d(a + t), d[0] = d(a - 1)
    __shared__ unsigned char taken[kTile];
    __shared__ int left[kPathLevels + 1], anc[kPathLevels + 1];  // ancestors of the first body from earlier
                                                                 // tiles, of the last body from any
    __shared__ int wmin[kTile / 32], listed[2];
    __shared__ unsigned levels;  // bit l: cells of level l start in the tile
    if (build_off(s.ctrl)) return;  // grid-uniform: only earlier kernels set either
    const int n = s.n, root = n + s.cap;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const unsigned below = (1u << lane) - 1u;
    const int a = blockIdx.x * kTile, m = min(kTile, n - a), i = a + t;
    if (t < 2) listed[t] = 0;
    if (t == 0) levels = 0;
    if (i < n) {
        const int body = s.sorted[i];
        key_sh[t] = path[i];
        base_sh[t] = b.base[i];
        node[t] = body;
        pm[t] = s.body_cur[body];
    }
    cnt_sh[t] = 1;
    taken[t] = 0;
    if constexpr (kQuad)
        for (int k = 0; k < 6; ++k) q6[k][t] = 0.0f;
    __syncthreads();
    int own = -1;
    if (i + 1 < n && i < n) own = common_levels(key_sh[t], t + 1 < m ? key_sh[t + 1] : path[i + 1]);
    d[t + 1] = (signed char)own;
    item[t] = (own + 1) << 16 | t;
    if (t == 0) d[0] = a > 0 ? (signed char)common_levels(path[a - 1], key_sh[0]) : (signed char)-1;
    __syncthreads();
    const int pre = d[t], lo = max(pre, 0);
    const unsigned some = __reduce_or_sync(0xffffffffu, own > lo ? (2u << own) - (2u << lo) : 0u);
    if (lane == 0 && some) atomicOr(&levels, some);
    // shallowest common level of the tile's bodies up to this one and the body before the tile
    int shallow = pre;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, shallow, o);
        if (lane >= o) shallow = min(shallow, u);
    }
    if (lane == 31) wmin[w] = shallow;
    if (w == 1 && lane >= 1 && lane <= (int)d[0]) {  // a level per lane
        // at the levels of the regions their table has the answer, below them
        // the bounds of the search
        int from = 0, m0 = a;
        if (b.levels) {
            const int r = region_of(key_sh[0], b.levels), sh = 3 * max(b.levels - lane, 0);
            from = b.start[r >> sh << sh];
            if (lane <= b.levels) m0 = from + 1;
        }
        const int st = from + first_sharing([&](int k) { return path[from + k]; }, m0 - from, key_sh[0], lane);
        const int pst = st > 0 ? common_levels(path[st - 1], path[st]) : 0;
        left[lane] = cell_number(b.base[st], pst, lane);
    }
    // the tile's own cells, deepest level first
    const int j = t & 7;
    const unsigned group = 0xffu << (lane & 24);
    __syncthreads();
    int turn = 0;
    for (unsigned todo = levels; todo;) {
        const int l = 31 - __clz(todo);
        todo &= ~(1u << l);
        turn ^= 1;
        const bool mine = i < n && lo < l && l <= own;
        const unsigned mk = __ballot_sync(0xffffffffu, mine);
        int at = 0;
        if (lane == 0 && mk) at = atomicAdd(&listed[turn], __popc(mk));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (mine) list[at + __popc(mk & below)] = (short)t;
        __syncthreads();  // also: the items of the level below are in place
        const int cells = listed[turn];
        if (t == 0) listed[turn ^ 1] = 0;
        for (int g = t >> 3; g < cells; g += kTile / 8) {
            const int st = list[g];
            int f = st, nch = 0, k = st, end;
            bool inside = false;
            do {  // the children's first places
                if (nch == j) f = k;
                ++nch;
                end = item[k];
                inside = (end >> 16) - 1 < l;
                k = (end & 0xffff) + 1;
            } while (!inside && k < m && nch < 8);
            // (more than eight items: those of a child that reaches beyond the tile)
            if (!inside) continue;
            const int cell = cell_number(base_sh[st], max((int)d[st], 0), l), c = cell - n;
            const bool have = j < nch;
            const float4 p = pm[f];
            const int id = node[f], o = octant_at(key_sh[f], l);
            const CellSums sums = sum_children(group, (1u << nch) - 1u, p, cnt_sh[f]);
            const unsigned used = __reduce_or_sync(group, have ? 1u << o : 0u);
            s.wchild[c * 8 + j] = have ? id : kEmpty;
            s.wpm[c * 8 + j] = have ? p : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (!((used >> j) & 1u)) s.child[c * 8 + j] = kEmpty;
            if (have) s.child[c * 8 + o] = id;
            float q[6];
            if constexpr (kQuad) {
#pragma unroll
                for (int x = 0; x < 6; ++x) q[x] = q6[x][f];
                s.wqa[c * 8 + j] = make_float4(q[0], q[1], q[2], q[3]);
                s.wqb[c * 8 + j] = make_float2(q[4], q[5]);
                sum_quadrupoles(group, (1u << nch) - 1u, p, sums, q);
            }
            if (have && j > 0) taken[f] = 1;
            __syncwarp(group);  // the items are read before the first one becomes the cell
            if (j == 0) {
                const float4 v = make_float4(sums.X, sums.Y, sums.Z, sums.M);
                s.count[c] = sums.cnt;
                s.start[c] = 0;  // complete
                s.cell_pm[c] = v;
                pm[st] = v;
                node[st] = cell;
                cnt_sh[st] = sums.cnt;
                item[st] = end;
                if constexpr (kQuad) {
                    s.cell_q[2 * c] = make_float4(q[0], q[1], q[2], q[3]);
                    s.cell_q[2 * c + 1] = make_float4(q[4], q[5], 0.0f, 0.0f);
                    for (int x = 0; x < 6; ++x) q6[x][st] = q[x];
                }
            }
        }
        __syncthreads();
    }
    __syncthreads();
    for (int k = 0; k < w; ++k) shallow = min(shallow, wmin[k]);
    if (w == 0) {
        const int end = d[m];
        bool here = false;
        if (lane >= 1 && lane <= end) {
            const int st = first_sharing([&](int k) { return key_sh[k]; }, m, key_sh[m - 1], lane);
            here = d[st] < lane;
            anc[lane] = here ? cell_number(base_sh[st], max((int)d[st], 0), lane) : left[lane];
        }
        __syncwarp();
        if (here) {
            const int p = lane > 1 ? anc[lane - 1] : root;
            s.child[(p - n) * 8 + octant_at(key_sh[m - 1], lane - 1)] = anc[lane];
            s.parent[anc[lane] - n] = p;
        }
    }
    __syncthreads();
    if (i < n && !taken[t]) {
        const int p = max(max(pre, (item[t] >> 16) - 1), 0);  // level of the parent
        const int parent = p == 0 ? root : (shallow >= p ? left[p] : anc[p]);
        s.child[(parent - n) * 8 + octant_at(key_sh[t], p)] = node[t];
    }
}

// ---------------------------------------------------------------------------
// k_top: the cells that reach over a tile's edge, the root among them.  Each is
// completed by whichever eight lanes bring its arrival counter to the number
// of its children.  Or, when the step takes the insertions:
// all of the build, the summarisation and the sort, with barriers over the
// grid, which is no larger than what is resident.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool grid_barrier(Ctrl *c, int *arrived, int target) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(arrived, 1);
        ok = 1;
        for (long long spins = 0; ld_volatile(arrived) < target;) {
            if (++spins > kSpinCap) {
                set_status(c, kStSpinTimeout, target);
                ok = 0;
                break;
            }
            __nanosleep(64);
        }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

constexpr int kTopThreads = 512;
// cell `cell` by eight lanes: lane j holds octant slot j's child ch (mask: the
// slots that have one), complete in memory
template <bool kQuad>
__device__ __forceinline__ void top_cell(const DevSim &s, int cell, int ch, unsigned mask, unsigned group, int j) {
    const int n = s.n, c = cell - n;
    const bool have = ch >= 0;
    float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int cnt = 1;
    float q[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (have && ch < n) p = s.body_cur[ch];
    if (ch >= n) {
        p = __ldcg(&s.cell_pm[ch - n]);
        cnt = __ldcg(&s.count[ch - n]);
        if constexpr (kQuad) {
            const float4 oa = __ldcg(&s.cell_q[2 * (ch - n)]), ob = __ldcg(&s.cell_q[2 * (ch - n) + 1]);
            q[0] = oa.x;
            q[1] = oa.y;
            q[2] = oa.z;
            q[3] = oa.w;
            q[4] = ob.x;
            q[5] = ob.y;
        }
    }
    // children first, in slot order, then empty places
    const int rank = __popc(mask & ((1u << j) - 1u));
    const int at = c * 8 + (have ? rank : __popc(mask) + j - rank);
    s.wchild[at] = have ? ch : kEmpty;
    s.wpm[at] = p;
    const CellSums sums = sum_children(group, mask, p, cnt);
    if constexpr (kQuad) {
        s.wqa[at] = make_float4(q[0], q[1], q[2], q[3]);
        s.wqb[at] = make_float2(q[4], q[5]);
        sum_quadrupoles(group, mask, p, sums, q);
    }
    if (j == 0) {
        s.count[c] = sums.cnt;
        s.cell_pm[c] = make_float4(sums.X, sums.Y, sums.Z, sums.M);
        if constexpr (kQuad) {
            s.cell_q[2 * c] = make_float4(q[0], q[1], q[2], q[3]);
            s.cell_q[2 * c + 1] = make_float4(q[4], q[5], 0.0f, 0.0f);
        }
    }
}

template <bool kQuad>
__global__ void __launch_bounds__(kTopThreads, 1) k_top(DevSim s, BuildScratch b) {
    wait_for_previous();
    Ctrl *ctrl = s.ctrl;
    const int n = s.n, root = n + s.cap;
    const int first = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    if (!ctrl->insert) {  // grid-uniform: only earlier kernels set it
        if (read_status(ctrl)) return;
        const int cells = b.ctl[kBuildTop];
        const int j = threadIdx.x & 7;
        const unsigned group = 0xffu << (threadIdx.x & 24);
        for (int k = first >> 3; k < cells; k += stride >> 3) {
            int cell = b.top[k];
            int ch = s.child[(cell - n) * 8 + j];
            unsigned mask = (__ballot_sync(group, ch >= 0) >> (threadIdx.x & 24)) & 0xffu;
            // children that were complete before this kernel
            const int ready = __popc(__ballot_sync(group, ch >= 0 && (ch < n || s.start[ch - n] == 0)));
            int arrivals = ready;
            while (arrivals > 0) {
                if (arrivals != __popc(mask)) {
                    int old = 0;
                    if (j == 0) old = atomicAdd(&s.arrive[cell - n], arrivals);
                    if (__shfl_sync(group, old, 0, 8) + arrivals != __popc(mask)) break;
                    __threadfence();
                }
                // the parent's row is on its way while the cell is summed
                const int up = cell == root ? root : s.parent[cell - n];
                const int up_ch = s.child[(up - n) * 8 + j];
                top_cell<kQuad>(s, cell, ch, mask, group, j);
                if (cell == root) break;
                cell = up;
                ch = up_ch;
                mask = (__ballot_sync(group, ch >= 0) >> (threadIdx.x & 24)) & 0xffu;
                __threadfence();  // this lane's stores before the arrival
                __syncwarp(group);
                arrivals = 1;
            }
        }
        return;
    }
    const int blocks = gridDim.x;
    // cells that k_cells numbered before it met equal paths are dropped
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ctrl->bottom = root;
        ctrl->max_depth = 0;
    }
    if (!grid_barrier(ctrl, &b.ctl[kBuildBarrier], blocks)) return;
    if (!read_status(ctrl)) {
        float box[6];
        load_box(ctrl, box);
        const GeoCube root_g = GeoCube::root(box);
        const long long cap = tree_spin_cap(ctrl);
        int deep = 0;
        for (int i = first; i < n; i += stride) {
            const int depth = insert_body<GeoCube, false>(s, root_g, i, cap);
            if (depth < 0) break;
            deep = max(deep, depth);
        }
        if (deep > 0) atomicMax(&ctrl->max_depth, deep);
    }
    if (!grid_barrier(ctrl, &b.ctl[kBuildBarrier], 2 * blocks)) return;
    const bool good = read_status(ctrl) == 0;
    const int bottom = ctrl->bottom;
    if (good)
        for (int k = bottom + first; k <= root; k += stride) summarize_from<kQuad>(s, k);
    if (!grid_barrier(ctrl, &b.ctl[kBuildBarrier], 3 * blocks) || !good) return;
    const long long cap = tree_spin_cap(ctrl);
    for (int k = root - first; k >= bottom; k -= stride)
        if (!sort_cell(s, k, cap)) return;
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
size_t build_scratch_ints(int n, int sm_count) {
    const size_t regions = (size_t)1 << (3 * build_levels(n));
    return kBuildCtl + kScanBlocks + (size_t)6 * 4 * sm_count + build_top_cells(n) + 2 * regions + 4;
}

BuildScratch build_scratch(int n, int sm_count, int *mem, void *keys16, void *ints12) {
    BuildScratch b{};
    b.levels = build_levels(n);
    const size_t regions = (size_t)1 << (3 * b.levels);
    b.ctl = mem;  // 16-byte aligned, as are the tables behind it
    b.total = b.ctl + kBuildCtl;
    b.count = b.total + kScanBlocks;
    b.start = b.count + regions;
    b.top = b.start + regions + 4;
    b.box = reinterpret_cast<unsigned *>(b.top + build_top_cells(n));
    b.path = static_cast<u64 *>(keys16);
    b.placed = b.path + n;
    b.rank = static_cast<int *>(ints12);
    b.who = b.rank + n;
    b.base = b.who + n;
    (void)sm_count;
    return b;
}

cudaError_t launch_tree_box(const DevSim &s, const BuildScratch &b, int sm_count, cudaStream_t st) {
    const int blocks = std::max(1, std::min(4 * sm_count, (s.n + 255) / 256));
    k_box<<<blocks, 256, 0, st>>>(s, b);  // not early: see launch.cuh
    return cudaGetLastError();
}

cudaError_t launch_tree_cells(const DevSim &s, const BuildScratch &b, int sm_count, cudaStream_t st, int *launches) {
    const int all = (s.n + 255) / 256;
    const int blocks = std::min(all, 8 * sm_count);
    cudaError_t e = launch_next(k_path, blocks, 256, st, s, b);
    if (b.levels) {
        const int per = scan_chunks(b.levels) * kScanRegions;
        if (e == cudaSuccess)
            e = launch_next(k_scan, ((1 << (3 * b.levels)) + per - 1) / per, kScanThreads, st, s, b);
        if (e == cudaSuccess) e = launch_next(k_place, blocks, 256, st, s, b);
        if (e == cudaSuccess) e = launch_next(k_rank, all, 256, st, s, b);
    } else {
        if (e == cudaSuccess) e = launch_next(k_rank_all, (s.n + 31) / 32, 32 * kRankWarps, st, s, b);
    }
    if (e == cudaSuccess)
        e = launch_next(k_cells, (s.n + kCellBodies - 1) / kCellBodies, kTile, st, s, b, b.levels ? b.path : b.placed);
    *launches = b.levels ? 5 : 3;
    return e;
}

cudaError_t launch_tree_sums(const DevSim &s, const BuildScratch &b, int quadrupole, int sm_count, cudaStream_t st) {
    const int tiles = (s.n + kTile - 1) / kTile;
    const u64 *path = b.levels ? b.path : b.placed;
    cudaError_t e = launch_next(quadrupole ? k_link<true> : k_link<false>, tiles, kTile, st, s, b, path);
    if (e == cudaSuccess) e = launch_next(quadrupole ? k_top<true> : k_top<false>, sm_count, kTopThreads, st, s, b);
    return e;
}

}  // namespace nbgb
