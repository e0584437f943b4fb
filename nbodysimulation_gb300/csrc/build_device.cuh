// build_device.cuh -- the per-tile work of the build from sorted octant paths
// as device functions, shared by the kernels of a single system (k_build.cu)
// and those that walk a table of systems (k_batch_build.cu).
#pragma once
#include <type_traits>

#include "bh_device.cuh"

namespace nbgb {

typedef unsigned long long u64;
constexpr int kPathLevels = 21;
constexpr int kTile = 256;          // sorted bodies per block of k_cells and k_link, one per thread

// ---------------------------------------------------------------------------
// paths
// ---------------------------------------------------------------------------
// (RefBox: the slot of the super-root is 0 for every body)
template <class Geo>
__device__ __forceinline__ u64 octant_path(Geo g, const float4 P, int levels) {
    u64 key = 0;
#pragma unroll
    for (int l = 0; l < levels; ++l) {
        key = key * 8 + (u64)g.octant(P.x, P.y, P.z);
        g.descend(P.x, P.y, P.z);
    }
    return key;
}
// region of a path: its first b.levels levels (behind the one that all bodies
// share with the reference's tree semantics)
__device__ __forceinline__ int region_of(u64 key, const BuildScratch &b) {
    return (int)(key >> (3 * (kPathLevels - b.levels - b.ref)));
}
// levels two paths share: the level of the deepest cell that holds both
__device__ __forceinline__ int common_levels(u64 a, u64 b) {
    const u64 x = a ^ b;
    return x ? (__clzll((long long)x) - 1) / 3 : kPathLevels;
}
__device__ __forceinline__ int octant_at(u64 key, int level) { return (int)(key >> (3 * (kPathLevels - 1 - level))) & 7; }
__device__ __forceinline__ bool build_off(const Ctrl *c) { return read_status(c) != 0 || c->insert != 0; }

// Crowded regions: a block ranks its bodies against all of their regions, at 20 to
// 60 ns a body there, which the insertions beat from some number of bodies in one
// region on, the larger the system the later, or when the system has more than
// kPairsPerBody pairs a body.  (Normal positions and one body far out, ms up to the
// sums, insertions / ranking, by the most bodies in a region: 4,000 of 4,000 0.14 /
// 0.14; 3,433 of 20,000 0.17 / 0.29, 6,089 0.17 / 0.41; 4,047 of 30,011 0.18 / 0.30;
// 8,402 of 262,144 0.39 / 0.60; 4,870 of 1,000,003 0.83 / 0.70.)  With the
// reference's semantics, whose boxes part bodies later, a system that is all in one
// region mostly inserts in the end (3,000 bodies 0.15, ranked first 0.22).
constexpr int kCrowd = 2048;
constexpr int kPairsPerBody = 4096;
__device__ __forceinline__ int crowd_limit(int n, int ref) {
    return !ref && n <= 2 * kCrowd ? n : kCrowd + (n >> 6);
}

// Path of body i; its region and its place there.  One body too many in a region
// sends the step to the insertions (it alone: a store by every body behind it took
// 0.3 ms).
template <class Geo>
__device__ __forceinline__ void path_body(const DevSim &s, const BuildScratch &b, const Geo &root, int i) {
    constexpr int kLevels = std::is_same<Geo, RefBox>::value ? kPathLevels - 1 : kPathLevels;
    const u64 key = octant_path<Geo>(root, s.body_cur[i], kLevels);
    b.path[i] = key;
    if (b.levels) {
        // a warp whose bodies are all in one region (nearly every one when a body
        // is far out) adds once: 60,000 bodies 0.36 -> 0.32 ms a step
        const int r = region_of(key, b), lane = threadIdx.x & 31;
        const unsigned active = __activemask();
        const int first = __ffs(active) - 1;
        int at = 0;
        if (__all_sync(active, r == __shfl_sync(active, r, first))) {
            if (lane == first) at = atomicAdd(&b.count[r], __popc(active));
            at = __shfl_sync(active, at, first) + __popc(active & ((1u << lane) - 1u));
        } else {
            at = atomicAdd(&b.count[r], 1);
        }
        b.rank[i] = at;
        if (at == crowd_limit(s.n, b.ref)) s.ctrl->insert = 1;
    }
}

// Body i into its region.
__device__ __forceinline__ void place_body(const BuildScratch &b, int i) {
    const u64 key = b.path[i];
    const int at = b.start[region_of(key, b)] + b.rank[i];
    b.placed[at] = key;
    b.who[at] = i;
}

// Place of every body among those of its region: the number of smaller paths
// there, equal ones in the order they lie.  A block's regions lie end to end and
// pass through shared memory.  Equal paths (21 levels do not part the bodies)
// end up side by side, where k_cells sees them.
constexpr int kRankChunk = 1024;
__device__ __forceinline__ void rank_tile(const DevSim &s, const BuildScratch &b, int tile) {
    __shared__ u64 sh[kRankChunk];
    const int first = tile * kTile, last = min(s.n, first + kTile) - 1;
    const int i = first + threadIdx.x;
    const u64 key = b.placed[min(i, last)];
    const int r = region_of(key, b);
    const int lo = b.start[r], hi = i < s.n ? b.start[r + 1] : lo;
    const int block_lo = b.start[region_of(b.placed[first], b)];
    const int block_hi = b.start[region_of(b.placed[last], b) + 1];
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
__device__ __forceinline__ void cells_tile(const DevSim &s, const BuildScratch &b, const u64 *path, int tile) {
    __shared__ u64 key_sh[kCellBodies + 2];  // the paths of bodies a - 1 .. a + kCellBodies
    __shared__ int base_sh[kCellBodies];
    __shared__ int warp_tot[32];
    __shared__ int first, deepest;
    if (__syncthreads_or(build_off(s.ctrl))) return;  // an overflow elsewhere stops whole blocks
    Ctrl *c = s.ctrl;
    const int t = threadIdx.x, n = s.n, a = tile * kCellBodies, m = min(kCellBodies, n - a);
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
                const int at = atomicAdd(&b.ctl[kBuildTop], 1);  // completed by k_top
                b.top[at] = cell;
                s.start[k] = 1 + at;
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
__device__ __forceinline__ void link_tile(const DevSim &s, const BuildScratch &b, const u64 *path, int tile) {
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
    const int a = tile * kTile, m = min(kTile, n - a), i = a + t;
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
            const int r = region_of(key_sh[0], b), sh = 3 * max(b.levels + b.ref - lane, 0);
            from = b.start[r >> sh << sh];
            if (lane <= b.levels + b.ref) m0 = from + 1;
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
// The cells that reach over a tile's edge, the root among them: each is
// completed by whichever eight lanes bring its arrival counter to the number
// of its children.
// ---------------------------------------------------------------------------
// The data of child ch (a body or a complete cell).
template <bool kQuad>
__device__ __forceinline__ void load_child(const DevSim &s, int ch, float4 &p, int &cnt, float (&q)[6]) {
    const int n = s.n;
    p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    cnt = 1;
#pragma unroll
    for (int k = 0; k < 6; ++k) q[k] = 0.0f;
    if (ch >= 0 && ch < n) p = s.body_cur[ch];
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
}

// cell `cell` by eight lanes: lane j holds octant slot j's child ch and its data
// (mask: the slots that have one); q: the child's moments in, the cell's out
template <bool kQuad>
__device__ __forceinline__ CellSums finish_cell(const DevSim &s, int cell, int ch, unsigned mask, unsigned group, int j,
                                                const float4 p, int cnt, float (&q)[6]) {
    const int c = cell - s.n;
    const bool have = ch >= 0;
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
    return sums;
}

// A short list in one block: every cell's row in shared memory, where a finished
// cell is entered, so a level costs the sums and no round trips to L2 (which
// take 2.5 us, six or seven levels deep).  Longer lists keep one block too long.
// The sums of both kernels, by the arrival counters in memory / here (GB300, us):
// monopoles, 3,000 bodies 37 / 27, 6,007 38 / 31, 12,000 40 / 34, 20,000 (340
// cells) 41 / 41; quadrupoles, 3,000 bodies 39 / 33, 12,000 (190 cells) 48 / 51.
constexpr int kTopSharedBodies = 1 << 15;  // beyond, a list is longer anyhow (20 cells per 1,024 bodies)
template <bool kQuad>
constexpr int kTopShared = kQuad ? 128 : 256;
template <bool kQuad>
struct TopShared {
    float4 pm[kTopShared<kQuad>][8];
    int cnt[kTopShared<kQuad>][8], id[kTopShared<kQuad>][8];
    float q[kQuad ? kTopShared<kQuad> : 1][6][8];
    int cell[kTopShared<kQuad>];     // ~cell: all children were complete before this kernel
    int up[kTopShared<kQuad>];       // 8 * place of the parent + slot there
    int pending[kTopShared<kQuad>];  // children still to come
};
template <bool kQuad, int kThreads>
__device__ __forceinline__ void top_cells_shared(const DevSim &s, const BuildScratch &b, int cells,
                                                 TopShared<kQuad> &sh) {
    const int n = s.n, j = threadIdx.x & 7, groups = kThreads >> 3;
    const unsigned group = 0xffu << (threadIdx.x & 24);
    // all of a group's cells at once: three trips to L2 in a row
    constexpr int kRounds = kTopShared<kQuad> * 8 / kThreads;
    int cell[kRounds], ch[kRounds], at[kRounds];  // at: 1 + the child's place in the list
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const int k = (threadIdx.x >> 3) + r * groups;
        cell[r] = k < cells ? b.top[k] : -1;
    }
#pragma unroll
    for (int r = 0; r < kRounds; ++r) ch[r] = cell[r] >= 0 ? s.child[(cell[r] - n) * 8 + j] : kEmpty;
#pragma unroll
    for (int r = 0; r < kRounds; ++r) at[r] = ch[r] >= n ? s.start[ch[r] - n] : 0;
    float4 p[kRounds];
    int cnt[kRounds];
    float q[kRounds][6];
#pragma unroll
    for (int r = 0; r < kRounds; ++r) load_child<kQuad>(s, at[r] > 0 ? kEmpty : ch[r], p[r], cnt[r], q[r]);
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const int k = (threadIdx.x >> 3) + r * groups;
        if (cell[r] < 0) break;
        sh.pm[k][j] = p[r];
        sh.cnt[k][j] = cnt[r];
        sh.id[k][j] = ch[r];
        if constexpr (kQuad)
            for (int x = 0; x < 6; ++x) sh.q[k][x][j] = q[r][x];
        if (at[r] > 0) sh.up[at[r] - 1] = 8 * k + j;
        const int open = __popc(__ballot_sync(group, at[r] > 0));
        if (j == 0) {
            sh.cell[k] = open ? cell[r] : ~cell[r];
            sh.pending[k] = open;
        }
    }
    __syncthreads();
    for (int k = threadIdx.x >> 3; k < cells; k += groups) {
        if (sh.cell[k] >= 0) continue;
        for (int c = k;;) {
            const int cell = c == k ? ~sh.cell[c] : sh.cell[c], ch = sh.id[c][j];
            const unsigned mask = (__ballot_sync(group, ch >= 0) >> (threadIdx.x & 24)) & 0xffu;
            float q[6];
            if constexpr (kQuad)
#pragma unroll
                for (int x = 0; x < 6; ++x) q[x] = sh.q[c][x][j];
            const CellSums sums = finish_cell<kQuad>(s, cell, ch, mask, group, j, sh.pm[c][j], sh.cnt[c][j], q);
            if (c == 0) break;  // the root
            const int up = sh.up[c], parent = up >> 3, slot = up & 7;
            int left = 0;
            if (j == 0) {
                sh.pm[parent][slot] = make_float4(sums.X, sums.Y, sums.Z, sums.M);
                sh.cnt[parent][slot] = sums.cnt;
                if constexpr (kQuad)
#pragma unroll
                    for (int x = 0; x < 6; ++x) sh.q[parent][x][slot] = q[x];
                __threadfence_block();
                left = atomicSub(&sh.pending[parent], 1);
                __threadfence_block();
            }
            if (__shfl_sync(group, left, 0, 8) != 1) break;
            __syncwarp(group);
            c = parent;
        }
    }
}

// cells first, first + stride, .. of the list, eight lanes each
template <bool kQuad>
__device__ __forceinline__ void top_cells(const DevSim &s, const BuildScratch &b, int cells, int first, int stride) {
    const int n = s.n, root = n + s.cap;
    const int j = threadIdx.x & 7;
    const unsigned group = 0xffu << (threadIdx.x & 24);
    for (int k = first; k < cells; k += stride) {
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
            float4 p;
            int cnt;
            float q[6];
            load_child<kQuad>(s, ch, p, cnt, q);
            finish_cell<kQuad>(s, cell, ch, mask, group, j, p, cnt, q);
            if (cell == root) break;
            cell = up;
            ch = up_ch;
            mask = (__ballot_sync(group, ch >= 0) >> (threadIdx.x & 24)) & 0xffu;
            __threadfence();  // this lane's stores before the arrival
            __syncwarp(group);
            arrivals = 1;
        }
    }
}

}  // namespace nbgb
