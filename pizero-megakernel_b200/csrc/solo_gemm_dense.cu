// Instantiations of the single-operator GEMM for BF16 and FP8 operands.
#include "solo_gemm.cuh"

namespace pi0 {
cudaError_t launch_solo_gemm_dense(const SoloGemm& p, int cg, int grid, size_t smem, cudaStream_t stream) {
    const int form = (p.g.operands * 8 + p.g.epilogue) * 4 + cg;
    switch (form) {
        case (GEMM_BF16 * 8 + EPI_F32) * 4 + 1: return launch_solo_gemm_form<GEMM_BF16, EPI_F32, 1>(p, grid, smem, stream);
        case (GEMM_BF16 * 8 + EPI_F32) * 4 + 2: return launch_solo_gemm_form<GEMM_BF16, EPI_F32, 2>(p, grid, smem, stream);
        case (GEMM_BF16 * 8 + EPI_BF16) * 4 + 1: return launch_solo_gemm_form<GEMM_BF16, EPI_BF16, 1>(p, grid, smem, stream);
        case (GEMM_BF16 * 8 + EPI_BF16) * 4 + 2: return launch_solo_gemm_form<GEMM_BF16, EPI_BF16, 2>(p, grid, smem, stream);
        case (GEMM_FP8 * 8 + EPI_F32) * 4 + 1: return launch_solo_gemm_form<GEMM_FP8, EPI_F32, 1>(p, grid, smem, stream);
        case (GEMM_FP8 * 8 + EPI_F32) * 4 + 2: return launch_solo_gemm_form<GEMM_FP8, EPI_F32, 2>(p, grid, smem, stream);
        case (GEMM_FP8 * 8 + EPI_BF16) * 4 + 1: return launch_solo_gemm_form<GEMM_FP8, EPI_BF16, 1>(p, grid, smem, stream);
        case (GEMM_FP8 * 8 + EPI_BF16) * 4 + 2: return launch_solo_gemm_form<GEMM_FP8, EPI_BF16, 2>(p, grid, smem, stream);
        default: return cudaErrorNotSupported;
    }
}

int solo_gemm_clusters(int ctas) {
    static int known[64][9] = {};
    int device = 0, n = 0;
    if (ctas == 1) return 1 << 20;                           // (bounded by the workers)
    if (ctas > 8 || cudaGetDevice(&device) != cudaSuccess) return 0;
    if (device < 64 && known[device][ctas]) return known[device][ctas];
    const auto kernel = pi0_gemm_kernel<GEMM_FP8, EPI_F32, 2>;
    const size_t smem = kSoloDataBytes + kSoloCtlBytes + 1024;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = ctas;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(ctas * 64);
    config.blockDim = dim3(128 + 32 * solo_drain_warps(GEMM_FP8, EPI_F32));
    config.dynamicSmemBytes = smem;
    config.attrs = &attr;
    config.numAttrs = 1;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &config) != cudaSuccess)
        n = 0;
    if (device < 64) known[device][ctas] = n;
    return n;
}
}  // namespace pi0
