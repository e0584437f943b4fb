// k_build.cu -- bounding box, octree, centres of mass and in-order sort of a
// single system, from sorted octant paths: with the cubic root or, up to
// kRefPathBodies, the reference's boxes and super-root.
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

#include "build_device.cuh"
#include "launch.cuh"

namespace nbgb {

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
    if (threadIdx.x < 8) b.ctl[kBuildPhases + threadIdx.x] = 0;
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
        b.ctl[kBuildScan] = 0;
        b.ctl[kBuildTop] = 1;
        b.top[0] = s.n + s.cap;
        *reinterpret_cast<u64 *>(&b.ctl[kBuildPairs]) = 0;
    }
}

__global__ void __launch_bounds__(256) k_path(DevSim s, BuildScratch b) {
    wait_for_previous();
    if (build_off(s.ctrl)) return;
    float box[6];
    load_box(s.ctrl, box);
    const int first = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    for (int i = first; i < s.n; i += stride) {
        if (i > first && ld_volatile(&s.ctrl->insert)) return;  // a crowded region: the paths are of no use
        if (b.ref) path_body(s, b, RefBox::root(box), i);
        else path_body(s, b, GeoCube::root(box), i);
    }
}

// Exclusive scan of the region counts: a block adds up the totals of the
// blocks before it as they appear.  The blocks, at most kScanBlocks with as many
// chunks of kScanRegions each as that needs, take their places in the order in
// which they start, so one waits only for blocks that run.  Clears the counts for
// the next step and adds up the pairs that ranking the regions will compare.  No
// block leaves early: the counts must be zero before the next step, also when a
// wait gives up (a step that failed before this kernel counted nothing).
inline __host__ __device__ int scan_chunks(int levels) {
    const int chunks = ((1 << (3 * levels)) + kScanRegions - 1) / kScanRegions;
    return (chunks + kScanBlocks - 1) / kScanBlocks;
}
__global__ void __launch_bounds__(kScanThreads, 2) k_scan(DevSim s, BuildScratch b) {
    wait_for_previous();
    __shared__ int warp_tot[32];
    __shared__ u64 warp_sq[32];
    __shared__ int before, place;
    if (threadIdx.x == 0) place = gridDim.x > 1 ? atomicAdd(&b.ctl[kBuildScan], 1) : 0;
    __syncthreads();
    const int regions = 1 << (3 * b.levels), chunks = scan_chunks(b.levels);
    const int begin = place * chunks * kScanRegions;
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
    if (threadIdx.x == 0) st_volatile(&b.total[place], total + 1);
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
        for (int k = threadIdx.x; k < place; k += 32) {
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
    if (place == 0 && threadIdx.x == 0) b.start[regions] = s.n;
}
__device__ __forceinline__ bool too_crowded(const DevSim &s, const BuildScratch &b) {
    return *reinterpret_cast<const volatile u64 *>(&b.ctl[kBuildPairs]) > (u64)s.n * kPairsPerBody;
}

__global__ void __launch_bounds__(256) k_place(DevSim s, BuildScratch b) {
    wait_for_previous();
    if (build_off(s.ctrl) || too_crowded(s, b)) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < s.n; i += gridDim.x * blockDim.x) place_body(b, i);
}

__global__ void __launch_bounds__(kTile) k_rank(DevSim s, BuildScratch b) {
    wait_for_previous();
    if (__syncthreads_or(build_off(s.ctrl))) return;  // other blocks of this kernel may set `insert`
    if (too_crowded(s, b)) {                          // grid-uniform
        s.ctrl->insert = 1;
        return;
    }
    rank_tile(s, b, blockIdx.x);
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

__global__ void __launch_bounds__(kTile) k_cells(DevSim s, BuildScratch b, const u64 *path) {
    wait_for_previous();
    cells_tile(s, b, path, blockIdx.x);
}

// kBlocks: least resident blocks per SM.  Five (48 registers) fill one another's
// barriers where the tiles are two waves or more; else the compiler's choice (80 and 58)
// (the sums, four / five blocks, ms: 4M with quadrupoles 0.705 / 0.646, 500,000
// 0.092 / 0.084, 100,003 with quadrupoles 0.0579 / 0.0585; six 0.659 at 4M; four
// asked for, 0.785: another schedule).
template <bool kQuad, int kBlocks>
__global__ void __launch_bounds__(kTile, kBlocks) k_link(DevSim s, BuildScratch b, const u64 *path) {
    wait_for_previous();
    link_tile<kQuad>(s, b, path, blockIdx.x);
}

// ---------------------------------------------------------------------------
// k_top: the cells that reach over a tile's edge, the root among them.  Each is
// completed by whichever eight lanes bring its arrival counter to the number
// of its children.  Or, when the step takes the insertions: all of the build,
// the summarisation and the sort, as phases (run_phase).
// ---------------------------------------------------------------------------
template <bool kQuad, int kThreads>
__global__ void __launch_bounds__(kThreads, 1) k_top(DevSim s, BuildScratch b, bool may_share) {
    wait_for_previous();
    Ctrl *ctrl = s.ctrl;
    const int n = s.n, root = n + s.cap;
    const int first = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    if (!ctrl->insert) {  // grid-uniform: only earlier kernels set it
        if (read_status(ctrl)) return;
        extern __shared__ __align__(16) unsigned char top_smem[];
        const int cells = b.ctl[kBuildTop];
        if (!may_share || cells > kTopShared<kQuad>) top_cells<kQuad>(s, b, cells, first >> 3, stride >> 3);
        else if (blockIdx.x == 0) top_cells_shared<kQuad, kThreads>(s, b, cells, *reinterpret_cast<TopShared<kQuad> *>(top_smem));
        return;
    }
    const int t = threadIdx.x;
    int *phases = b.ctl + kBuildPhases;
    const auto gave_up = [&]() {
        if (t == 0) set_status(ctrl, kStSpinTimeout, 0);
    };
    // cells that k_cells numbered before it met equal paths are dropped
    if (!run_phase(phases, 1, [&](int) {
            if (t > 0) return;
            ctrl->bottom = root;
            ctrl->max_depth = 0;
        }))
        return gave_up();
    float box[6];
    load_box(ctrl, box);
    const long long cap = tree_spin_cap(ctrl);
    int deep = 0;
    if (!run_phase(phases + 2, (n + kThreads - 1) / kThreads, [&](int chunk) {
            const int i = chunk * kThreads + t;
            if (i >= n || read_status(ctrl)) return;
            deep = max(deep, b.ref ? insert_body<RefBox, true>(s, RefBox::root(box), i, cap)
                                   : insert_body<GeoCube, false>(s, GeoCube::root(box), i, cap));
            if (deep > 0) atomicMax(&ctrl->max_depth, deep);
        }))
        return gave_up();
    if (read_status(ctrl)) return;  // grid-uniform: the insertions are over
    const int bottom = ld_volatile(&ctrl->bottom), chunks = (root - bottom) / kThreads + 1;
    if (!run_phase(phases + 4, chunks, [&](int chunk) {
            const int k = bottom + chunk * kThreads + t;
            if (k <= root) summarize_from<kQuad>(s, k);
        }))
        return gave_up();
    if (!run_phase(phases + 6, chunks, [&](int chunk) {
            const int k = bottom + chunk * kThreads + t;
            if (k <= root) sort_bodies_of(s, k);
        }))
        gave_up();
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
size_t build_scratch_ints(int n, int sm_count) {
    const size_t regions = (size_t)1 << (3 * build_levels(n));
    return kBuildCtl + kScanBlocks + (size_t)6 * 4 * sm_count + build_top_cells(n) + 2 * regions + 4;
}

BuildScratch build_scratch(int n, int ref, int *mem, void *keys16, void *ints12) {
    BuildScratch b{};
    b.ref = ref;
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
    const auto link = tiles >= 8 * sm_count ? (quadrupole ? k_link<true, 5> : k_link<false, 5>)
                                            : (quadrupole ? k_link<true, 1> : k_link<false, 1>);
    cudaError_t e = launch_next(link, tiles, kTile, st, s, b, path);
    // shared memory only where the list may be short: the SMs' split of it would
    // hold back the walk's blocks
    const bool may_share = s.n <= kTopSharedBodies;
    const size_t shared = !may_share ? 0 : quadrupole ? sizeof(TopShared<true>) : sizeof(TopShared<false>);
    // 1,024 threads a block where the list's groups fill them many times over (the
    // sums with 512 / 1,024 threads, ms: 12,000 bodies with quadrupoles 0.049 /
    // 0.054, 100,003 0.058 / 0.061, 262,144 0.0627 / 0.0640, 4M 0.643 / 0.600)
    const int threads = s.n >= (1 << 20) ? 1024 : 512;
    const auto top = threads == 1024 ? (quadrupole ? k_top<true, 1024> : k_top<false, 1024>)
                                     : (quadrupole ? k_top<true, 512> : k_top<false, 512>);
    if (e == cudaSuccess && shared)
        e = cudaFuncSetAttribute(top, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
    if (e == cudaSuccess) e = launch_next_shared(top, sm_count, threads, shared, st, s, b, may_share);
    return e;
}

}  // namespace nbgb
