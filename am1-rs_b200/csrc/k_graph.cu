// Control kernels of the captured SCF solve (CUDA graph with device-side loops).
//
// The graph path runs a whole batched solve as one graph launch: the SCF iterations are the body
// of a conditional WHILE node, and inside it the purification steps are the body of a second one.
// These single-thread kernels decide, on the device, whether a loop goes round again, so the host
// reads nothing until the solve is done.  Each loop carries its own counter, and a loop ends when
// the counter reaches its cap whatever the other conditions say: the SCF loop after max_scf
// iterations, the purification loop after max_steps products, exactly as the host-driven loop of
// the eager path is bounded.
#include <cuda_runtime.h>

#include "kernels.h"

namespace am1 {

// Before the SCF loop: iteration counter and total-step counter to 0, the loop armed when any
// iteration is allowed at all.
__global__ void k_scf_arm(cudaGraphConditionalHandle h, GraphLoop* loop, int max_scf) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    loop->scf_iter = 0;
    loop->sp2_total = 0;
    loop->stalled = 0;
    cudaGraphSetConditional(h, max_scf > 0 ? 1u : 0u);
}

// Before each purification loop: its step counter and the counters of the step's update
// (k_sp2_update_cond, which decides the loop) to 0, the loop armed.
__global__ void k_sp2_arm(cudaGraphConditionalHandle h, GraphLoop* loop) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    loop->sp2_step = 0;
    loop->sp2_active = 0;
    loop->ticket = 0;
    cudaGraphSetConditional(h, 1u);
}

// After each SCF iteration (k_converge has counted the molecules still iterating in active[0]): go round
// again while any is and fewer than max_scf iterations were done, unless some purification stalled
// (need_eigen[-1]): those molecules wait for the host, which runs their eigensolver.
__global__ void k_scf_cond(cudaGraphConditionalHandle h, GraphLoop* loop, const int* active, const int* need_eigen, int max_scf) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const int it = loop->scf_iter + 1, stalled = need_eigen[-1] != 0;
    loop->scf_iter = it;
    loop->stalled = stalled;
    cudaGraphSetConditional(h, (active[0] > 0 && it < max_scf && !stalled) ? 1u : 0u);
}

}  // namespace am1
