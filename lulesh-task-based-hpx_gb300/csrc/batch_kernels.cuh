// Batched persistent phase kernels, shared by every arithmetic variant.
//
// Included at the end of a variant's translation unit (after its
// forces_elem / nodes_node / kinematics_elem / material_elem). One launch
// per phase covers every active instance of a batch: a fixed grid of blocks
// pulls (instance, tile) items from a per-phase queue counter until the
// queue is empty, so large and small instances, and material tiles with 1 or
// 20 EOS passes, share the SMs without a launch per instance. Material tiles
// are queued most expensive first.
//
// A block takes `grab` consecutive tiles per queue access, copies a tile's
// Mesh (device pointers of that instance) into shared memory when the
// instance changes, and runs the variant's per-element function over the
// tile. The force, node and kinematics phases fetch their next queue position
// while the current tiles run (their tiles cost alike, so the reservation
// costs no balance); the material phase takes its next position only when
// its tiles are done, so that its cost-sorted queue stays dynamically
// balanced (reserving ahead cost 4-6 % of a serving run).
//
// The bounds (kBatchBlocks, blocks of kBatchMaxBlock per SM by phase) keep the
// phases near the occupancy of the single-problem kernels: inlined into the
// tile loop the double forces and kinematics take 200 registers by
// themselves, which leaves 8 warps per SM. us per cycle of 14 problems of
// s=16-64, and of 10 of 18-40, with one block asked for and as given here:
// double 943, 498 -> 768, 344, mixed 570, 260 -> 548, 245; exact 18-40 2163
// -> 1459. More blocks cost spills (double material 3: 787, 4: 805; mixed
// material 4: 590; double kinematics 3: 832).
// Each instance keeps its own dt (DevTime), and the material phase lowers
// the instance's Courant/hydro minima with atomic minima on the doubles' bit
// patterns (exact for positive values, so the order does not matter).

namespace lulesh {
namespace LULESH_VARIANT {

// Atomic min of a positive double, through its bit pattern (positive IEEE
// doubles order like their unsigned 64-bit patterns).
__device__ __forceinline__ void atomic_min_pos(double* addr, double v) {
    atomicMin(reinterpret_cast<unsigned long long*>(addr),
              static_cast<unsigned long long>(__double_as_longlong(v)));
}

#if LULESH_EXACT
constexpr int kBatchBlocks[4] = {3, 4, 2, 3};  // forces, nodes, kinematics, material
#elif LULESH_FLOAT_Q
constexpr int kBatchBlocks[4] = {3, 4, 3, 3};
#else
constexpr int kBatchBlocks[4] = {2, 4, 2, 2};
#endif
template <int PHASE>
__global__ void __launch_bounds__(kBatchMaxBlock, kBatchBlocks[PHASE]) kb_phase(BatchCtl c, int grab) {
    constexpr int kind = (PHASE == 1) ? TILES_NODE : (PHASE == 3) ? TILES_MAT : TILES_ELEM;
    constexpr bool kPrefetch = PHASE != 3;
    __shared__ __align__(16) unsigned long long s_mesh[(sizeof(Mesh) + 7) / 8];
    __shared__ int s_tile;
    __shared__ int s_active;
    __shared__ double s_dt;
    const Mesh& m = *reinterpret_cast<const Mesh*>(s_mesh);
    const int ntiles = __ldg(c.ntiles + kind);
    const BatchTile* tiles = c.tiles[kind];
    int cur_inst = -1;
    if (threadIdx.x == 0) s_tile = (int)atomicAdd(&c.queue[PHASE], (unsigned)grab);
    __syncthreads();
    int t0 = s_tile;
    while (t0 < ntiles) {
        const int t1 = min(t0 + grab, ntiles);
        __syncthreads();  // every thread has read s_tile
        // the next queue position, fetched while this grab's tiles run
        if (kPrefetch && threadIdx.x == 0) s_tile = (int)atomicAdd(&c.queue[PHASE], (unsigned)grab);
        for (int t = t0; t < t1; ++t) {
            const BatchTile tile = tiles[t];
            if (tile.inst != cur_inst) {  // the same for every thread of the block
                __syncthreads();          // the previous instance's Mesh is no longer read
                const unsigned long long* src = reinterpret_cast<const unsigned long long*>(c.meshes + tile.inst);
                for (int k = threadIdx.x; k < (int)((sizeof(Mesh) + 7) / 8); k += blockDim.x) s_mesh[k] = src[k];
                if (threadIdx.x == 0) {
                    s_active = c.times[tile.inst].active;
                    s_dt = c.times[tile.inst].deltatime;
                }
                __syncthreads();
                cur_inst = tile.inst;
            }
            if (!s_active) continue;
            if (PHASE == 3) {
                DtMin<LULESH_EXACT> dt;
                const MatClass cls{tile.first, tile.count, tile.lanes, 0};
                const int per_warp = 32 / cls.lanes;
                for (int w = threadIdx.x >> 5; w * per_warp < cls.count; w += blockDim.x >> 5) {
                    int pos, r;
                    material_place(cls, w, pos, r);
                    material_elem<true>(m, pos, r, cls.lanes, dt);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    dt.dtc = fmin(dt.dtc, __shfl_down_sync(0xffffffffu, dt.dtc, o));
                    dt.dth = fmin(dt.dth, __shfl_down_sync(0xffffffffu, dt.dth, o));
                }
                if ((threadIdx.x & 31) == 0) {
                    atomic_min_pos(&m.result->dtcourant, dt.dtc);
                    atomic_min_pos(&m.result->dthydro, dt.dth);
                }
            } else {
                for (int k = threadIdx.x; k < tile.count; k += blockDim.x) {
                    if (PHASE == 0) forces_elem(m, tile.first + k);
                    if (PHASE == 2) kinematics_elem(m, tile.first + k, s_dt);
                    if (PHASE == 1) nodes_node(m, tile.first + k, s_dt);
                }
            }
        }
        if (!kPrefetch && threadIdx.x == 0) s_tile = (int)atomicAdd(&c.queue[PHASE], (unsigned)grab);
        __syncthreads();  // thread 0's next queue position is visible
        t0 = s_tile;
    }
}

int launch_batch_phase(int phase, const BatchCtl& c, const BatchLaunch& l, cudaStream_t s) {
    switch (phase) {
        case 0: kb_phase<0><<<l.grid, l.block, 0, s>>>(c, l.grab); break;
        case 1: kb_phase<1><<<l.grid, l.block, 0, s>>>(c, l.grab); break;
        case 2: kb_phase<2><<<l.grid, l.block, 0, s>>>(c, l.grab); break;
        default: kb_phase<3><<<l.grid, l.block, 0, s>>>(c, l.grab); break;
    }
    return 1;
}

int batch_occupancy(int phase, int block) {
    int n = 0;
    cudaError_t e;
    switch (phase) {
        case 0: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kb_phase<0>, block, 0); break;
        case 1: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kb_phase<1>, block, 0); break;
        case 2: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kb_phase<2>, block, 0); break;
        default: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kb_phase<3>, block, 0); break;
    }
    return e == cudaSuccess ? n : 0;
}

}  // namespace LULESH_VARIANT
}  // namespace lulesh
