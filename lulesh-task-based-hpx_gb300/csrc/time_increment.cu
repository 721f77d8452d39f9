// Device-side time control for the CUDA-graph forms of the time loop.
// Built with --fmad=false, as the host TimeIncrement is built without
// contraction; time_advance.cuh rounds alike either way, as the material
// kernels compile it too.
#include "time_advance.cuh"

namespace lulesh {

// Single problem, one thread: the first cycle's step. The material kernel's
// last block advances the others (finish_dt_reduction).
__global__ void k_time_increment(DevTime* t, const StepResult* r) {
    advance_time(t, r);
}

// Batch: one thread per slot; re-arms the slot's dt minima (1e20, as
// lulesh.cc:2214-2215) and clears the per-phase tile queues.
__global__ void kb_time_increment(BatchCtl c) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0)
        for (int k = 0; k < 4; ++k) c.queue[k] = 0u;
    if (i >= c.slots) return;
    if (advance_time(c.times + i, c.results + i)) {
        c.results[i].dtcourant = 1.0e+20;
        c.results[i].dthydro = 1.0e+20;
    }
}

__global__ void kb_time_finish(BatchCtl c) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.slots) return;
    if (c.times[i].active) finish_time(c.times + i, c.results + i);
}

int launch_time_increment(DevTime* t, StepResult* r, cudaStream_t s) {
    k_time_increment<<<1, 1, 0, s>>>(t, r);
    return 1;
}

int launch_batch_time_increment(const BatchCtl& c, cudaStream_t s) {
    kb_time_increment<<<blocks_for(c.slots, 128), 128, 0, s>>>(c);
    return 1;
}

int launch_batch_time_finish(const BatchCtl& c, cudaStream_t s) {
    kb_time_finish<<<blocks_for(c.slots, 128), 128, 0, s>>>(c);
    return 1;
}

}  // namespace lulesh
