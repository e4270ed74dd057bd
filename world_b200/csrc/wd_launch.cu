// wd_launch.cu -- device-side launches of the Verlet-list build's CUDA graphs.
//
// In a list-mode semi-implicit Euler step the contact kernel decides at its end
// whether the lists must be rebuilt before the next step. A conditional node after it
// costs about 8 us of device time per step even when not taken; instead, one thread
// of a one-block kernel tail-launches the build's device-launchable graph only when the
// decision says so (the launched graph runs after the step's graph has completed, and
// the next step's graph waits for it). The same kind of kernel takes the radix path where
// the search wants it: the mover path's kernels stand in the graph that holds the search's
// head, gated, and its last kernel launches the graph that sorts all keys instead. (A graph
// of its own for the mover path too cost its launch, 4 us, on every searched step and
// build.) After the listing it launches the steps that a chain has left.
//
// This is the only translation unit compiled with relocatable device code (the device
// runtime's cudaGraphLaunch): elsewhere -rdc would put the device ABI on the contact
// kernels and raise their spills.
#include "wd_kernels.h"

namespace wd {
namespace {

// Launches a graph behind the one that runs, and notes why it could not.
__device__ void tail_launch(cudaGraphExec_t graph, volatile uint32_t* failed) {
    const cudaError_t e =
        graph == nullptr ? cudaErrorInvalidResourceHandle : cudaGraphLaunch(graph, cudaStreamGraphTailLaunch);
    if (e != cudaSuccess) *failed = static_cast<uint32_t>(e);
}

__global__ void k_graph_if(const uint32_t* __restrict__ flag, cudaGraphExec_t graph,
                           volatile uint32_t* __restrict__ failed) {
    if (threadIdx.x != 0 || *flag == 0u) return;
    tail_launch(graph, failed);
}

__global__ void k_graph_chain(const uint32_t* __restrict__ ctrl, int steps, cudaGraphExec_t even,
                              cudaGraphExec_t odd, volatile uint32_t* __restrict__ failed) {
    if (threadIdx.x != 0 || ctrl[kLcDecision] == 0u) return;
    // the step that decided: the chain's steps before it are done, kLcLeft wait
    const int step = steps - 1 - static_cast<int>(ctrl[kLcLeft]);
    tail_launch(step & 1 ? odd : even, failed);
}

__global__ void k_build_end(uint32_t* __restrict__ ctrl, const cudaGraphExec_t* __restrict__ by_left,
                            const int* __restrict__ radix_flag, cudaGraphExec_t radix,
                            volatile uint32_t* __restrict__ failed) {
    if (threadIdx.x != 0) return;
    if (radix_flag != nullptr && *radix_flag != 0) {
        tail_launch(radix, failed);
    } else if (by_left != nullptr) {
        const uint32_t left = ctrl[kLcLeft];
        ctrl[kLcPending] = 0u;
        ctrl[kLcLeft] = 0u;
        // steps that nothing takes up (no handle) are an error, not steps left out
        if (left > 0u) tail_launch(by_left[left], failed);
    }
}

}  // namespace

void launch_graph_chain(const uint32_t* list_ctrl, int steps, cudaGraphExec_t even,
                        cudaGraphExec_t odd, volatile uint32_t* failed, cudaStream_t st) {
    k_graph_chain<<<1, 32, 0, st>>>(list_ctrl, steps, even, odd, failed);
}

void launch_build_end(uint32_t* list_ctrl, const cudaGraphExec_t* by_left, const int* radix_flag,
                      cudaGraphExec_t radix, volatile uint32_t* failed, cudaStream_t st) {
    k_build_end<<<1, 32, 0, st>>>(list_ctrl, by_left, radix_flag, radix, failed);
}

void launch_graph_if(const uint32_t* flag, cudaGraphExec_t graph, volatile uint32_t* failed,
                     cudaStream_t st) {
    k_graph_if<<<1, 32, 0, st>>>(flag, graph, failed);
}

}  // namespace wd
