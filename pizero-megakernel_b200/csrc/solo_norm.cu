// LayerNorm / RMSNorm launched by itself: the rows of op_norm.cuh, two warps per row, in a kernel of their own.
//
// What bounds it is a chain, not a rate: one trip for the rows, their statistics, the quantiser, one trip back - 1.8 us - and 1.2 us from the
// end of one launch to the release of the next.  The next launch is let in at once: CTAs of 256 threads without dynamic shared memory find room
// beside these, and wait.  51 x 1024 to NVFP4, back to back: 3.3 us, most of which is the host's call (as a program of one stage 5.1); 768 x
// 2048: 5.1 (10.3).
#include "op_norm.cuh"
#include "solo.h"

namespace pi0 {

__global__ void __launch_bounds__(512) pi0_norm_kernel(const __grid_constant__ SoloNorm p) {
    __shared__ float red[2 * 16];
    const NormParams& n = p.n;
    const int warp = threadIdx.x >> 5, group = warp >> 3, local_row = (warp & 7) >> 1;
    const int rows_per_block = static_cast<int>(blockDim.x) >> 6;
    grid_dependency_wait();
    grid_launch_dependents();
    // (norm weights next to the input rows, not behind their statistics)
    for (int i = threadIdx.x; i < (n.width * 4 + 127) >> 7; i += blockDim.x) {
        if (n.gamma) prefetch_l1(n.gamma + i * 32);
        if (n.beta) prefetch_l1(n.beta + i * 32);
    }
    for (int row0 = blockIdx.x * rows_per_block; row0 < n.rows; row0 += gridDim.x * rows_per_block) {
        const int row = row0 + group * kNormPairRows + local_row;
        norm_row_pair<false>(n, row, local_row, warp & 1, row < n.rows, red + group * 16);
        if (threadIdx.x == 0) atomicAdd(p.guard.counters + (row0 >> 7), 1u);
        if (row0 + static_cast<int>(gridDim.x) * rows_per_block < n.rows) __syncthreads();   // `red` is used again
    }
}

cudaError_t launch_solo_norm(const SoloNorm& p, int grid, int groups, cudaStream_t stream) {
    cudaLaunchAttribute serial{};
    serial.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    serial.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(grid);
    config.blockDim = dim3(256 * groups);
    config.stream = stream;
    config.attrs = &serial;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, pi0_norm_kernel, p);
}

}  // namespace pi0
