// k_force.cu -- the single-system Barnes-Hut force kernel: warps take
// groups of 32 sorted bodies from a global counter and walk the tree
// (force_group, force_device.cuh), then integrate.
#include "force_device.cuh"
#include "launch.cuh"

namespace nbgb {

// kBlocks: the launch bound that the registers follow.  Eight blocks per SM (128
// registers), or nine (96) where the groups fill the GPU more than twice over.
// What is resident follows from the shared memory too: of monopoles ten blocks with
// 96 registers, whose extra warps hide more of the walk than its tighter schedule
// costs; of compensated quadrupoles eight either way (27 KB a block), where the
// schedule itself is the faster one.  With quadrupoles and without compensation
// neither is (GB300, the walk in ms, bound eight / nine: monopoles, ball, 6,007
// bodies 0.0635 / 0.0657, 131,072 0.207 / 0.207, 200,000 0.290 / 0.287, 262,144
// 0.365 / 0.353, 1,000,000 1.303 / 1.246; quadrupoles compensated, 200,000 0.522 /
// 0.515, 4,194,304 11.78 / 11.57; quadrupoles, 1,000,000 1.305 / 1.310).
constexpr int kFewGroups = 8, kManyGroups = 9;
template <int kMethod, bool kComp, bool kEpsZero, bool kQuad, int kBlocks>
__global__ void __launch_bounds__(kForceThreads, kBlocks) k_force(DevSim s, StepParams p) {
    wait_for_previous();
    __shared__ float s_dq[kMaxDepth];
    __shared__ WarpLists<kQuad> s_lists[kForceWarps];
    __shared__ int s_skip, s_room;
    Ctrl *ctrl = s.ctrl;
    const int n = s.n;
    if (threadIdx.x == 0) {
        int skip = read_status(ctrl);
        if (!skip && ctrl->max_depth >= kMaxDepth) {
            set_status(ctrl, kStDepth, ctrl->max_depth);
            skip = 1;
        }
        s_skip = skip;
        s_room = stack_room(ctrl->max_depth);  // once a block: the line is busy with the counters
        float box[6];
        load_box(ctrl, box);
        make_thresholds(box, p.theta, p.eps, p.crit_ref, s_dq);
    }
    __syncthreads();
    if (s_skip) {  // a failed step keeps the step-start state
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
            s.body_next[i] = s.body_cur[i];
        return;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int ngroups = (n + 31) >> 5;
    while (true) {
        int g = 0;
        if (lane == 0) g = atomicAdd(&ctrl->work, 1);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= ngroups) break;
        force_group<kMethod, kComp, kEpsZero, kQuad>(s, p, s_dq, s_room, g, lane, s_lists[w]);
    }
}

template <int kMethod, bool kComp, bool kQuad, int kBlocks>
static cudaError_t launch_force_b(const DevSim &s, const StepParams &p, int sm_count, cudaStream_t st) {
    const bool ez = !(p.eps > 0.0f);
    const auto kernel = ez ? k_force<kMethod, kComp, true, kQuad, kBlocks> : k_force<kMethod, kComp, false, kQuad, kBlocks>;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kForceThreads, 0) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    int blocks = per_sm * sm_count;
    const int need = ((s.n + 31) / 32 + kForceWarps - 1) / kForceWarps;
    if (blocks > need) blocks = need > 0 ? need : 1;
    if (blocks == per_sm * sm_count) return launch_next(kernel, blocks, kForceThreads, st, s, p);
    kernel<<<blocks, kForceThreads, 0, st>>>(s, p);  // a part of the GPU: spread evenly (launch.cuh)
    return cudaGetLastError();
}

template <int kMethod, bool kComp, bool kQuad>
static cudaError_t launch_force_t(const DevSim &s, const StepParams &p, int sm_count, cudaStream_t st) {
    if constexpr (!kQuad || kComp)
        if ((s.n + 31) / 32 >= 2 * kFewGroups * kForceWarps * sm_count)
            return launch_force_b<kMethod, kComp, kQuad, kManyGroups>(s, p, sm_count, st);
    return launch_force_b<kMethod, kComp, kQuad, kFewGroups>(s, p, sm_count, st);
}

template <int kMethod>
static cudaError_t launch_force_m(const DevSim &s, const StepParams &p, int compensated, int sm_count,
                                  cudaStream_t st) {
    if (p.quadrupole) {
        return compensated ? launch_force_t<kMethod, true, true>(s, p, sm_count, st)
                           : launch_force_t<kMethod, false, true>(s, p, sm_count, st);
    }
    return compensated ? launch_force_t<kMethod, true, false>(s, p, sm_count, st)
                       : launch_force_t<kMethod, false, false>(s, p, sm_count, st);
}

cudaError_t launch_force(const DevSim &s, const StepParams &p, int compensated, int sm_count, cudaStream_t st) {
    switch (p.method) {
    case 1: return launch_force_m<1>(s, p, compensated, sm_count, st);
    case 2: return launch_force_m<2>(s, p, compensated, sm_count, st);
    case 3: return launch_force_m<3>(s, p, compensated, sm_count, st);
    default: return launch_force_m<0>(s, p, compensated, sm_count, st);
    }
}

}  // namespace nbgb
