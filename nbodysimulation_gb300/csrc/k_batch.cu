// k_batch.cu -- one launch per stage for many independent systems of uneven
// N.  Every kernel walks the batch's table of systems (SysDesc): the work
// of all systems is laid end to end in one index space per stage (bodies in
// chunks or tiles, warp groups, direct-sum target blocks) and a warp finds its
// system in the stage's prefix table.
// Barnes-Hut systems run the same per-item code as the single-system kernels;
// their trees are k_batch_build.cu's.  Small systems take the direct sum
// (direct_device.cuh).  A step is: box, paths, places, ranks, cells, sums in
// tiles, sums above, insertions, force, direct, flip -- captured once into a CUDA
// graph by the host.
#include <string>

#include "collide_device.cuh"
#include "direct_device.cuh"
#include "force_device.cuh"

namespace nbgb {

// ---------------------------------------------------------------------------
// force: warps take groups from one batch-wide counter; a warp recomputes its
// thresholds whenever its next group belongs to another system.  A system
// whose step failed keeps its step-start state.
// ---------------------------------------------------------------------------
// Shared memory of one warp of the batched force kernel.  The block has a
// runtime number of warps (TreeShape::force_warps), so the warps' records are
// laid out one after another in dynamic shared memory.
template <bool kQuad>
struct BatchForceWarp {
    float dq[kMaxDepth];
    WarpLists<kQuad> lists;
    // the current system's buffers and parameters: the walk reads them from
    // shared memory where the single-system kernel reads its kernel
    // parameters, instead of holding them in registers
    DevSim view;
    StepParams par;
    // the current system, its first group, its mode (0 walk, 1 keep the step-start
    // state of a failed step, 2 inert) and its stack_room: in shared memory, so
    // nothing of the outer loop stays live in registers during a walk
    int cur, begin, mode, room;
};
constexpr int kBatchForceMaxWarps = 8;

// Registers: 128 a thread (four blocks of four warps per SM), or 96 (five blocks)
// where monopole groups fill the GPU (kMany, launch_batch_force_t).
template <int kMethod, bool kComp, bool kQuad, bool kMany>
__global__ void __maxnreg__(kMany ? 96 : 128) k_batch_force(BatchTables t) {
    extern __shared__ __align__(16) unsigned char force_smem[];
    BatchForceWarp<kQuad> &me = reinterpret_cast<BatchForceWarp<kQuad> *>(force_smem)[threadIdx.x >> 5];
    float *const s_dq_w = me.dq;
    DevSim &s_view_w = me.view;
    StepParams &s_par_w = me.par;
    int &s_cur_w = me.cur, &s_begin_w = me.begin, &s_mode_w = me.mode;
    const int lane = threadIdx.x & 31;
    if (lane == 0) s_cur_w = -1;
    if (blockIdx.x == 0 && threadIdx.x > 0 && threadIdx.x < kBatchWorkInts) t.work[threadIdx.x] = 0;  // for the next step
    __syncwarp();
    while (true) {
        int gg = 0;
        if (lane == 0) gg = atomicAdd(t.work, 1);
        gg = __shfl_sync(0xffffffffu, gg, 0);
        if (gg >= t.groups) break;
        const int k = find_system(t.group_prefix, t.nsys, gg);
        if (k != s_cur_w) {
            __syncwarp();  // the previous system's view and thresholds are no longer read
            if (lane == 0) {
                const SysDesc &d = t.sys[k];
                const DevSim v = system_view(d);
                StepParams p = d.p;
                p.kdk_primed = v.ctrl->kdk_primed;
                s_view_w = v;
                s_par_w = p;
                int sk = 0;
                if (!system_live(v.ctrl)) {
                    sk = 2;
                } else if (read_status(v.ctrl)) {
                    sk = 1;
                } else if (v.ctrl->max_depth >= kMaxDepth) {
                    set_status(v.ctrl, kStDepth, v.ctrl->max_depth);
                    sk = 1;
                }
                float box[6];
                load_box(v.ctrl, box);
                make_thresholds(box, p.theta, p.eps, p.crit_ref, s_dq_w);
                s_cur_w = k;
                s_begin_w = d.group_begin;
                s_mode_w = sk;
                me.room = stack_room(v.ctrl->max_depth);
            }
            __syncwarp();
        }
        const int g = gg - s_begin_w;
        const int mode = s_mode_w;
        const DevSim &s = s_view_w;
        if (mode == 2) continue;
        if (mode == 1) {  // keep the step-start state
            const int i = g * 32 + lane;
            if (i < s.n) s.body_next[i] = s.body_cur[i];
            continue;
        }
        force_group<kMethod, kComp, false, kQuad>(s, s_par_w, s_dq_w, me.room, g, lane, me.lists);
    }
}

// ---------------------------------------------------------------------------
// direct: one block per 32 kI targets of one system, its kW warps sharing the
// system's bodies (direct_device.cuh); Plummer softening; fused integrator.  kI
// and kW come from the autotuner; a system's sums do not depend on them.
// ---------------------------------------------------------------------------
template <int kI, int kW>
__global__ void __launch_bounds__(32 * kW) k_batch_direct(BatchTables t) {
    __shared__ DirectShared<kI, kW> sh;
    const int k = find_system(t.dblock_prefix, t.nsys, blockIdx.x);
    const SysDesc &d = t.sys[k];
    if (!system_live(d.v.ctrl)) return;  // block-uniform, before any barrier
    const DevSim s = system_view(d);
    StepParams p = d.p;
    p.kdk_primed = s.ctrl->kdk_primed;
    const int n = s.n, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int base = (blockIdx.x - d.dblock_begin) * (32 * kI);
    direct_sum<kI, kW, false, kZeroAdds>(s.body_cur, n, 0, n, base, p.eps, warp, lane, sh);
    for (int q = threadIdx.x; q < 32 * kI; q += 32 * kW) {  // one round where kW >= kI
        const float3 a = direct_target_sum<kI, kW>(sh, q);
        const int i = base + q;
        if (i < n) integrate_any(s, p, i, s.body_cur[i], a.x * p.G, a.y * p.G, a.z * p.G);
    }
}

// ---------------------------------------------------------------------------
// flip: the next buffer becomes current; KDK systems are primed; one step
// of the system's budget is used
// ---------------------------------------------------------------------------
__global__ void k_batch_flip(BatchTables t) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= t.nsys) return;
    const SysDesc &d = t.sys[k];
    if (!d.active) return;
    Ctrl *c = d.v.ctrl;
    const int budget = c->budget;
    if (budget == 0) return;
    c->parity ^= 1;
    if (d.p.method == 3) c->kdk_primed = 1;
    if (budget > 0) c->budget = budget - 1;
}

// ---------------------------------------------------------------------------
// collision update of every system that asks for it (update_collision_local,
// kernels/collision_update.cl:17-83): one block per kCollideBlockBodies
// targets of one system (a tree system's in the order of its sort), the
// block form of the standalone kernel
// (collide_device.cuh), after the force and direct stages have integrated
// and before the flip (src/MyApp.cpp:593-596,606-610,622-625).  Systems with
// no steps left or a failed step are skipped.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kCollideThreads) k_batch_collision(BatchTables t) {
    const int k = find_system(t.cblock_prefix, t.nsys, blockIdx.x);
    const SysDesc &d = t.sys[k];
    if (!system_live(d.v.ctrl) || read_status(d.v.ctrl)) return;  // block-uniform, before any barrier
    const DevSim s = system_view(d);
    collide_block(s.body_next, s.vel, d.kind == kSysBH ? s.sorted : nullptr, s.n, s.n,
                  (blockIdx.x - d.cblock_begin) * kCollideThreads, s.ctrl);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
// Direct-sum variants the autotuner chooses from: {targets per lane, warps per
// block}.
struct DirectVariant {
    int ki, warps;
};
static const DirectVariant kDirectVariants[] = {{1, 4}, {1, 8}, {2, 4}, {2, 8}, {4, 4}, {4, 8},
                                                {1, 2}, {1, 1}, {2, 2}, {2, 1}, {4, 2}};
constexpr int kNumDirectVariants = sizeof(kDirectVariants) / sizeof(kDirectVariants[0]);
static_assert(kBatchDirectDefault < kNumDirectVariants, "the default is one of the variants");

int batch_direct_variants() { return kNumDirectVariants; }
std::string batch_direct_names() {  // "1w4.1w8. ...": targets per lane, warps
    std::string s;
    for (const DirectVariant &v : kDirectVariants)
        s += (s.empty() ? "" : ".") + std::to_string(v.ki) + "w" + std::to_string(v.warps);
    return s;
}
int batch_direct_block_bodies(int variant) { return 32 * kDirectVariants[variant].ki; }

static cudaError_t launch_direct_variant(const BatchTables &t, int variant, cudaStream_t st) {
    const int b = t.dblocks;
    switch (variant) {
    case 0: k_batch_direct<1, 4><<<b, 128, 0, st>>>(t); break;
    case 1: k_batch_direct<1, 8><<<b, 256, 0, st>>>(t); break;
    case 2: k_batch_direct<2, 4><<<b, 128, 0, st>>>(t); break;
    case 3: k_batch_direct<2, 8><<<b, 256, 0, st>>>(t); break;
    case 4: k_batch_direct<4, 4><<<b, 128, 0, st>>>(t); break;
    case 5: k_batch_direct<4, 8><<<b, 256, 0, st>>>(t); break;
    case 6: k_batch_direct<1, 2><<<b, 64, 0, st>>>(t); break;
    case 7: k_batch_direct<1, 1><<<b, 32, 0, st>>>(t); break;
    case 8: k_batch_direct<2, 2><<<b, 64, 0, st>>>(t); break;
    case 9: k_batch_direct<2, 1><<<b, 32, 0, st>>>(t); break;
    default: k_batch_direct<4, 2><<<b, 64, 0, st>>>(t); break;
    }
    return cudaGetLastError();
}

template <int kMethod, bool kComp, bool kQuad, bool kMany>
static cudaError_t launch_batch_force_b(const BatchTables &t, const TreeShape &shape, int sm_count,
                                        cudaStream_t st) {
    int warps = shape.force_warps;
    if (warps < 1 || warps > kBatchForceMaxWarps) warps = kForceWarps;
    const int threads = warps * 32;
    const size_t smem = sizeof(BatchForceWarp<kQuad>) * (size_t)warps;
    const void *fn = (const void *)k_batch_force<kMethod, kComp, kQuad, kMany>;
    if (smem > 48 * 1024) {  // beyond the default dynamic shared memory of a block: opt in
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    long long blocks = (long long)per_sm * sm_count * (shape.force_grid_pct > 0 ? shape.force_grid_pct : 100) / 100;
    const int need = (t.groups + warps - 1) / warps;
    if (blocks > need) blocks = need;
    if (blocks < 1) blocks = 1;
    k_batch_force<kMethod, kComp, kQuad, kMany><<<(int)blocks, threads, smem, st>>>(t);
    return cudaGetLastError();
}

// Sixteen warps per SM or more of groups: 96 registers (steps of monopole trees,
// GB300, ms, 128 / 96 registers: 18 of 20,000 bodies, 11,250 groups, 0.416 / 0.409;
// 512 of 3,000 1.20 / 1.15; 256 of 60,000 15.08 / 14.52; but 32 of 1,500, 1,500
// groups, 0.105 / 0.107 and 4 of 10,000 0.128 / 0.131).
template <int kMethod, bool kComp, bool kQuad>
static cudaError_t launch_batch_force_t(const BatchTables &t, const TreeShape &shape, int sm_count,
                                        cudaStream_t st) {
    if constexpr (!kQuad)
        if (t.groups >= 16 * sm_count) return launch_batch_force_b<kMethod, kComp, kQuad, true>(t, shape, sm_count, st);
    return launch_batch_force_b<kMethod, kComp, kQuad, false>(t, shape, sm_count, st);
}

template <int kMethod>
static cudaError_t launch_batch_force_m(const BatchTables &t, int comp, int quad, const TreeShape &shape,
                                        int sm_count, cudaStream_t st) {
    if (quad) return comp ? launch_batch_force_t<kMethod, true, true>(t, shape, sm_count, st)
                          : launch_batch_force_t<kMethod, false, true>(t, shape, sm_count, st);
    return comp ? launch_batch_force_t<kMethod, true, false>(t, shape, sm_count, st)
                : launch_batch_force_t<kMethod, false, false>(t, shape, sm_count, st);
}

// the tree stages and the force of every tree system; *launches gets the kernel count
static cudaError_t launch_batch_tree_stages(const BatchTables &t, int method, int comp, int quad,
                                            const TreeShape &shape, int sm_count, cudaStream_t st,
                                            int *launches) {
    cudaError_t e = cudaSuccess;
    int built = 0;
    if ((e = launch_batch_build(t, quad, sm_count, st, &built)) != cudaSuccess) return e;
    switch (method) {
    case 1: e = launch_batch_force_m<1>(t, comp, quad, shape, sm_count, st); break;
    case 2: e = launch_batch_force_m<2>(t, comp, quad, shape, sm_count, st); break;
    case 3: e = launch_batch_force_m<3>(t, comp, quad, shape, sm_count, st); break;
    default: e = launch_batch_force_m<0>(t, comp, quad, shape, sm_count, st); break;
    }
    if (launches) *launches = built + 1;
    return e;
}



// One batched step.  Kernels with no work in this batch are not launched.
// Returns the number of kernels launched through *launches.
cudaError_t launch_batch_step(const BatchTables &t, int method, int comp, int quad, int direct_variant,
                              const TreeShape &shape, int sm_count, cudaStream_t st, const StepFork *fork,
                              int *launches, bool advance) {
    int nl = 0;
    cudaError_t e = cudaSuccess;
    const int sb = (t.nsys + 127) / 128;
    const bool branch = fork && fork->aux && t.chunks > 0 && t.dblocks > 0;
    if (branch) {  // the direct sum beside the tree stages
        if ((e = cudaEventRecord(fork->fork, st)) != cudaSuccess ||
            (e = cudaStreamWaitEvent(fork->aux, fork->fork, 0)) != cudaSuccess ||
            (e = launch_direct_variant(t, direct_variant, fork->aux)) != cudaSuccess ||
            (e = cudaEventRecord(fork->join, fork->aux)) != cudaSuccess)
            return e;
        nl += 1;
    }
    if (t.chunks > 0) {
        int tl = 0;
        if ((e = launch_batch_tree_stages(t, method, comp, quad, shape, sm_count, st, &tl)) != cudaSuccess) return e;
        nl += tl;
    }
    if (branch && (e = cudaStreamWaitEvent(st, fork->join, 0)) != cudaSuccess) return e;
    if (t.dblocks > 0 && !branch) {
        if ((e = launch_direct_variant(t, direct_variant, st)) != cudaSuccess) return e;
        nl += 1;
    }
    if (!advance) {
        if (launches) *launches = nl;
        return cudaGetLastError();
    }
    if (t.cblocks > 0) {
        k_batch_collision<<<t.cblocks, kCollideThreads, 0, st>>>(t);
        nl += 1;
    }
    k_batch_flip<<<sb, 128, 0, st>>>(t);
    nl += 1;
    if (launches) *launches = nl;
    return cudaGetLastError();
}

__global__ void k_batch_clear(BatchTables t) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= t.nsys) return;
    Ctrl *c = t.sys[k].v.ctrl;
    c->status = 0;
    c->status_info = 0;
    c->interactions = 0;
    c->opened = 0;
    c->cell_interactions = 0;
}

cudaError_t launch_batch_clear(const BatchTables &t, cudaStream_t st) {
    k_batch_clear<<<(t.nsys + 127) / 128, 128, 0, st>>>(t);
    return cudaGetLastError();
}

}  // namespace nbgb
