// k_batch_build.cu -- boxes, trees, sums and sorts of a batch, from sorted octant
// paths: the stages of k_build.cu over all systems' tiles at once, with
// the tree semantics of each system.  A tree with bodies that 21 levels do not
// part, regions too crowded to rank, or the reference's semantics and more than
// kRefPathBodies bodies takes the insertions instead (ctrl->insert), all inside
// k_batch_insert.
//
// What bounds it: launches and chains of dependent L2 accesses, as for a single
// system; a batch's launches serve all its trees.  Top-level counts, top cells,
// insertions, summarisation by arrival counters and the sort by waits, with
// their boxes, took, against this (GB300, us a step): 5 trees of 56,000 bodies
// 207 -> 104, 18 of 320,000 243 -> 137; a step of 256 trees of 60,000 bodies 16.5
// -> 15.0 ms, and 9.8 -> 8.9 with the reference's semantics.
#include "build_device.cuh"
#include "launch.cuh"

namespace nbgb {

constexpr int kTileBlocks = kCellBodies / kTile;  // blocks of 256 bodies in an entry of tile_prefix
static_assert(kCellBodies == kBuildTileBodies, "k_batch_cells: one block per entry of tile_prefix");

// t.work: the force pass's counter, and the words of a step's insertions (zero
// between steps; two a phase)
enum { kWorkForce = 0, kWorkInsert = 1, kWorkPhases = 2 };
constexpr int kInsertPhases = 6;
static_assert(kWorkPhases + 2 * kInsertPhases <= kBatchWorkInts, "");

// A system's buffers while its tree is built.  The paths lie in the body buffer
// that the force pass writes next, the places in the regions where the sort
// will be, the chunks' boxes and then the bodies by region where the cells'
// numbers will be.
struct BuildSystem {
    DevSim s;
    BuildScratch b;
    int part;  // the block's part of the system
};
__device__ __forceinline__ BuildScratch scratch_of(const SysDesc &d, const DevSim &s) {
    BuildScratch b{};
    b.levels = d.build.levels;
    b.ref = d.p.tree_ref;
    b.ctl = d.build.mem;
    b.count = b.ctl + kBuildCtl;
    b.start = b.count + ((size_t)1 << (3 * b.levels));
    b.top = b.start + ((size_t)1 << (3 * b.levels)) + 4;
    b.base = b.top + build_top_cells(s.n);
    b.who = b.base;
    b.box = reinterpret_cast<unsigned *>(b.base);
    b.rank = s.sorted;
    b.path = reinterpret_cast<u64 *>(s.body_next);
    b.placed = b.path + s.n;
    return b;
}
// of block x of a grid with `per` blocks for every entry of tile_prefix
__device__ __forceinline__ BuildSystem build_system(const BatchTables &t, int x, int per) {
    const int tile = x / per, k = find_system(t.tile_prefix, t.nsys, tile);
    const SysDesc &d = t.sys[k];
    BuildSystem v;
    v.s = system_view(d);
    v.b = scratch_of(d, v.s);
    v.part = x - d.tile_begin * per;
    return v;
}
// (a system with no steps left is left alone; block-uniform where only earlier
// kernels set the words)
__device__ __forceinline__ bool left_alone(const Ctrl *c) { return !system_live(c) || build_off(c); }

// ---------------------------------------------------------------------------
// boxes (k_box, k_build.cu): one block per chunk of one system; the block that
// finishes a system's last chunk reduces the chunks' results and sets what its
// step starts from.  The blocks also clear the region counts.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_batch_box(BatchTables t) {
    __shared__ unsigned red[8][6];
    __shared__ int last;
    if (blockIdx.x == 0 && threadIdx.x == 0) t.work[kWorkForce] = 0;
    const SysDesc &d = t.sys[find_system(t.chunk_prefix, t.nsys, blockIdx.x)];
    const DevSim s = system_view(d);
    Ctrl *c = s.ctrl;
    if (!system_live(c)) return;  // block-uniform
    const BuildScratch b = scratch_of(d, s);
    const int chunks = (s.n + d.chunk - 1) / d.chunk, chunk = blockIdx.x - d.chunk_begin;
    int4 *count = reinterpret_cast<int4 *>(b.count);
    const int quads = 2 << (3 * (b.levels - 1));
    for (int q = chunk * blockDim.x + threadIdx.x; q < quads; q += chunks * blockDim.x)
        count[q] = make_int4(0, 0, 0, 0);
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
    for (int i = chunk * d.chunk + threadIdx.x; i < min(s.n, (chunk + 1) * d.chunk); i += blockDim.x) {
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
    unsigned r = block_reduce();
    if (chunks > 1) {
        unsigned *box = b.box;
        if (threadIdx.x < 6) {
            box[chunk * 6 + threadIdx.x] = r;
            __threadfence();
        }
        __syncthreads();
        if (threadIdx.x == 0) last = atomicAdd(&c->work, 1) == chunks - 1;
        __syncthreads();
        if (!last) return;
        __threadfence();
#pragma unroll
        for (int k = 0; k < 6; ++k) v[k] = k < 3 ? 0xFFFFFFFFu : 0u;
        for (int j = threadIdx.x; j < chunks; j += blockDim.x)
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                const unsigned x = __ldcg(&box[j * 6 + k]);
                v[k] = k < 3 ? min(v[k], x) : max(v[k], x);
            }
        r = block_reduce();
    }
    if (threadIdx.x < 6) c->bbox_key[threadIdx.x] = r;
    if (threadIdx.x < 8) s.child[s.cap * 8 + threadIdx.x] = kEmpty;
    if (threadIdx.x == 0) {
        c->bottom = s.n + s.cap;
        c->max_depth = 0;
        c->work = 0;  // chunks done
        c->insert = b.ref && s.n > kRefPathBodies;
        if (c->insert) t.work[kWorkInsert] = 1;
        s.arrive[s.cap] = 0;
        s.start[s.cap] = 0;
        s.count[s.cap] = 0;
        s.parent[s.cap] = -1;
        b.ctl[kBuildTop] = 1;  // the list of k_batch_top starts with the root
        b.top[0] = s.n + s.cap;
    }
}

// Start of every region of a system, by one block, kScanRegions at a time.
constexpr int kScanRegions = 8 * kTile;
__device__ __forceinline__ void scan_regions(const DevSim &s, const BuildScratch &b) {
    __shared__ int warp_tot[32];
    __shared__ u64 pairs;  // that ranking the regions will compare
    const int regions = 1 << (3 * b.levels);
    if (threadIdx.x == 0) pairs = 0;
    u64 sq = 0;
    int base = 0;
    for (int begin = 0; begin < regions; begin += kScanRegions) {
        const int at = begin + threadIdx.x * 8;
        int4 c0 = make_int4(0, 0, 0, 0), c1 = c0;
        if (at < regions) {
            c0 = __ldcg(reinterpret_cast<const int4 *>(&b.count[at]));
            c1 = __ldcg(reinterpret_cast<const int4 *>(&b.count[at]) + 1);
        }
        sq += (u64)c0.x * c0.x + (u64)c0.y * c0.y + (u64)c0.z * c0.z + (u64)c0.w * c0.w + (u64)c1.x * c1.x +
              (u64)c1.y * c1.y + (u64)c1.z * c1.z + (u64)c1.w * c1.w;
        int total;
        const int ex = block_exclusive_sum(c0.x + c0.y + c0.z + c0.w + c1.x + c1.y + c1.z + c1.w, warp_tot, &total);
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
            reinterpret_cast<int4 *>(&b.start[at])[0] = o0;
            reinterpret_cast<int4 *>(&b.start[at])[1] = o1;
        }
        base += total;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0 && sq) atomicAdd(&pairs, sq);
    __syncthreads();
    if (threadIdx.x == 0) {
        b.start[regions] = s.n;
        if (pairs > (u64)s.n * kPairsPerBody) s.ctrl->insert = 1;
    }
}

// paths; the block that finishes a system's last bodies scans its regions
__global__ void __launch_bounds__(kTile) k_batch_path(BatchTables t) {
    wait_for_previous();
    __shared__ int last;
    const BuildSystem v = build_system(t, blockIdx.x, kTileBlocks);
    const int blocks = (v.s.n + kTile - 1) / kTile;
    Ctrl *c = v.s.ctrl;
    // block-uniform: only earlier kernels set a status (`insert` may appear meanwhile)
    if (v.part >= blocks || !system_live(c) || read_status(c)) return;
    const int i = v.part * kTile + threadIdx.x;
    if (i < v.s.n && !ld_volatile(&c->insert)) {
        float box[6];
        load_box(c, box);
        if (v.b.ref) path_body(v.s, v.b, RefBox::root(box), i);
        else path_body(v.s, v.b, GeoCube::root(box), i);
    }
    __syncthreads();  // the block's counts are in (its atomics have returned)
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(&c->work, 1) == blocks - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x == 0) c->work = 0;
    if (ld_volatile(&c->insert)) return;  // every block has arrived
    scan_regions(v.s, v.b);
}

__global__ void __launch_bounds__(kTile) k_batch_place(BatchTables t) {
    wait_for_previous();
    const BuildSystem v = build_system(t, blockIdx.x, kTileBlocks);
    if (left_alone(v.s.ctrl)) return;
    const int i = v.part * kTile + threadIdx.x;
    if (i < v.s.n) place_body(v.b, i);
}

__global__ void __launch_bounds__(kTile) k_batch_rank(BatchTables t) {
    wait_for_previous();
    const BuildSystem v = build_system(t, blockIdx.x, kTileBlocks);
    if (v.part * kTile >= v.s.n || left_alone(v.s.ctrl)) return;  // block-uniform: only earlier kernels set either
    rank_tile(v.s, v.b, v.part);
}

__global__ void __launch_bounds__(kTile) k_batch_cells(BatchTables t) {
    wait_for_previous();
    const BuildSystem v = build_system(t, blockIdx.x, 1);
    if (!system_live(v.s.ctrl)) return;
    cells_tile(v.s, v.b, v.b.path, v.part);  // looks at the status and at `insert` itself
    __syncthreads();
    if (threadIdx.x == 0 && ld_volatile(&v.s.ctrl->insert)) t.work[kWorkInsert] = 1;
}

template <bool kQuad>
__global__ void __launch_bounds__(kTile) k_batch_link(BatchTables t) {
    wait_for_previous();
    const BuildSystem v = build_system(t, blockIdx.x, kTileBlocks);
    if (v.part * kTile >= v.s.n || !system_live(v.s.ctrl)) return;
    link_tile<kQuad>(v.s, v.b, v.b.path, v.part);
}

// ---------------------------------------------------------------------------
// insertions of the systems that take them (bh_device.cuh): top-level counts
// per chunk, top cells, insertions, the used cells laid end to end,
// summarisation and sort, as phases of one kernel (run_phase).  A step without
// insertions pays 2 us for it.  18 trees of 20,000 bodies, one far out in each:
// 0.64 ms a step, with a kernel per stage 0.65.
// ---------------------------------------------------------------------------
constexpr int kInsertThreads = 256;

__device__ __forceinline__ bool inserts(const SysDesc &d) {
    const Ctrl *c = d.v.ctrl;
    return d.active && d.kind == kSysBH && system_live(c) && !read_status(c) && c->insert;
}

// Bodies i0 + threadIdx.x .. of a system; its depth, or -1.
template <class Geo, bool kRef, bool kTop>
__device__ __forceinline__ int insert_chunk(const DevSim &s, const TopTables &top, int i0, int i1) {
    float box[6];
    load_box(s.ctrl, box);
    const Geo root_g = Geo::root(box);
    int deep = 0;
    const long long cap = tree_spin_cap(s.ctrl);
    for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
        int depth;
        if constexpr (kTop) depth = insert_from_top(s, top, root_g, i, cap);
        else depth = insert_body<Geo, kRef>(s, root_g, i, cap);
        if (depth < 0) return -1;
        deep = max(deep, depth);
    }
    return deep;
}

static_assert((1 << (3 * kBatchTopMaxLevels)) <= 32 * kInsertThreads, "top_cells_block: at most 32 regions a thread");
template <bool kQuad>
__global__ void __launch_bounds__(kInsertThreads, 4) k_batch_insert(BatchTables t) {
    wait_for_previous();
    if (!t.work[kWorkInsert]) return;  // grid-uniform: only earlier kernels set it
    __shared__ int bins[1 << (3 * kBatchTopMaxLevels)];
    __shared__ int warp_tot[32];
    const int tid = threadIdx.x;
    int *phases = t.work + kWorkPhases;
    const auto gave_up = [&]() {
        if (tid == 0)
            for (int k = 0; k < t.nsys; ++k)
                if (inserts(t.sys[k])) set_status(t.sys[k].v.ctrl, kStSpinTimeout, 0);
    };
    // top-level counts
    if (!run_phase(phases, t.chunks, [&](int x) {
            const SysDesc &d = t.sys[find_system(t.chunk_prefix, t.nsys, x)];
            if (!inserts(d)) return;  // block-uniform: nothing sets a status here
            const DevSim s = system_view(d);
            const int i0 = (x - d.chunk_begin) * d.chunk;
            if (tid == 0 && i0 == 0) {  // without the cells numbered before `insert` was set
                s.ctrl->bottom = s.n + s.cap;
                s.ctrl->max_depth = 0;
            }
            if (!d.top.levels) return;
            float box[6];
            load_box(s.ctrl, box);
            top_count_range(s, d.top, GeoCube::root(box), i0, min(s.n, i0 + d.chunk), blockDim.x, bins);
        }))
        return gave_up();
    // top cells: a block per system, whose status only it sets here
    if (!run_phase(phases + 2, t.nsys, [&](int k) {
            const SysDesc &d = t.sys[k];
            const bool mine = inserts(d) && d.top.levels;
            __syncthreads();
            if (mine) top_cells_block(system_view(d), d.top);
        }))
        return gave_up();
    // insertions
    if (!run_phase(phases + 4, t.chunks, [&](int x) {
            const SysDesc &d = t.sys[find_system(t.chunk_prefix, t.nsys, x)];
            if (!__shfl_sync(0xffffffffu, (int)inserts(d), 0)) return;  // a status may appear meanwhile
            const DevSim s = system_view(d);
            const int i0 = (x - d.chunk_begin) * d.chunk, i1 = min(s.n, i0 + d.chunk);
            const int depth = d.p.tree_ref     ? insert_chunk<RefBox, true, false>(s, d.top, i0, i1)
                              : d.top.levels ? insert_chunk<GeoCube, false, true>(s, d.top, i0, i1)
                                             : insert_chunk<GeoCube, false, false>(s, d.top, i0, i1);
            __syncwarp();
            const int deep = __reduce_max_sync(0xffffffffu, depth);
            if ((tid & 31) == 0 && deep > 0) atomicMax(&s.ctrl->max_depth, deep);
        }))
        return gave_up();
    // every tree's allocated cells [bottom, root], one after another
    if (!run_phase(phases + 6, 1, [&](int) {
            int carry = 0;
            for (int first = 0; first < t.nsys; first += blockDim.x) {
                const int k = first + tid;
                int used = 0;
                if (k < t.nsys && inserts(t.sys[k]))
                    used = t.sys[k].v.n + t.sys[k].v.cap - ld_volatile(&t.sys[k].v.ctrl->bottom) + 1;
                int total;
                const int before = carry + block_exclusive_sum(used, warp_tot, &total);
                if (k < t.nsys) t.used_prefix[k] = before;
                carry += total;
            }
            if (tid == 0) t.used_prefix[t.nsys] = carry;
        }))
        return gave_up();
    const int total = __ldcg(&t.used_prefix[t.nsys]), chunks = (total + kInsertThreads - 1) / kInsertThreads;
    int lo = 0, hi = 0, k = 0, first = 0, par = 0;  // the system of the last cell, its range, first cell and parity
    const auto locate = [&](int x) {
        if (x >= lo && x < hi) return;
        int a = 0, z = t.nsys;
        while (z - a > 1) {
            const int mid = (a + z) >> 1;
            if (__ldcg(&t.used_prefix[mid]) <= x) a = mid;
            else z = mid;
        }
        k = a;
        lo = __ldcg(&t.used_prefix[k]);
        hi = __ldcg(&t.used_prefix[k + 1]);
        first = ld_volatile(&t.sys[k].v.ctrl->bottom);
        par = system_parity(t.sys[k]);
    };
    if (!run_phase(phases + 8, chunks, [&](int chunk) {
            const int x = chunk * kInsertThreads + tid;
            if (x >= total) return;
            locate(x);
            summarize_from<kQuad>(system_view_par(t.sys[k], par), first + (x - lo));
        }))
        return gave_up();
    if (!run_phase(phases + 10, chunks, [&](int chunk) {
            const int x = chunk * kInsertThreads + tid;
            if (x >= total) return;
            locate(x);
            sort_bodies_of(t.sys[k].v, first + (x - lo));  // reads no body buffer
        }))
        gave_up();
}

constexpr int kTopThreads = 512;
template <bool kQuad>
__global__ void __launch_bounds__(kTopThreads) k_batch_top(BatchTables t) {
    wait_for_previous();
    extern __shared__ __align__(16) unsigned char top_smem[];
    const BuildSystem v = build_system(t, blockIdx.x, 1);
    if (left_alone(v.s.ctrl)) return;
    const int cells = v.b.ctl[kBuildTop];
    if (cells <= kTopShared<kQuad>) {
        if (v.part == 0) top_cells_shared<kQuad, kTopThreads>(v.s, v.b, cells, *reinterpret_cast<TopShared<kQuad> *>(top_smem));
        return;
    }
    // an entry of 1,024 bodies has about 20 of a system's cells, a block room for 64
    const int entries = (v.s.n + kBuildTileBodies - 1) / kBuildTileBodies;
    top_cells<kQuad>(v.s, v.b, cells, v.part * (kTopThreads / 8) + (threadIdx.x >> 3), entries * (kTopThreads / 8));
}

cudaError_t launch_batch_build(const BatchTables &t, int quadrupole, int sm_count, cudaStream_t st, int *launches) {
    k_batch_box<<<t.chunks, 256, 0, st>>>(t);
    cudaError_t e = cudaGetLastError();
    const int blocks = t.tiles * kTileBlocks;
    *launches = 1;
    if (blocks > 0) {
        if (e == cudaSuccess) e = launch_next(k_batch_path, blocks, kTile, st, t);
        if (e == cudaSuccess) e = launch_next(k_batch_place, blocks, kTile, st, t);
        if (e == cudaSuccess) e = launch_next(k_batch_rank, blocks, kTile, st, t);
        if (e == cudaSuccess) e = launch_next(k_batch_cells, t.tiles, kTile, st, t);
        if (e == cudaSuccess)
            e = launch_next(quadrupole ? k_batch_link<true> : k_batch_link<false>, blocks, kTile, st, t);
        const auto top = quadrupole ? k_batch_top<true> : k_batch_top<false>;
        const size_t shared = quadrupole ? sizeof(TopShared<true>) : sizeof(TopShared<false>);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(top, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
        if (e == cudaSuccess) e = launch_next_shared(top, t.tiles, kTopThreads, shared, st, t);
        *launches += 6;
    }
    const auto insert = quadrupole ? k_batch_insert<true> : k_batch_insert<false>;
    if (e == cudaSuccess) e = launch_next(insert, 4 * sm_count, kInsertThreads, st, t);
    *launches += 1;
    return e;
}

}  // namespace nbgb
