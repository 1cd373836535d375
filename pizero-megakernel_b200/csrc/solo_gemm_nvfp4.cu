// Instantiations of the single-operator GEMM for NVFP4 operands.
#include "solo_gemm.cuh"

namespace pi0 {
cudaError_t launch_solo_gemm_nvfp4(const SoloGemm& p, int cg, int grid, size_t smem, cudaStream_t stream) {
    switch (p.g.epilogue * 4 + cg) {
        case EPI_F32 * 4 + 1: return launch_solo_gemm_form<GEMM_NVFP4, EPI_F32, 1>(p, grid, smem, stream);
        case EPI_F32 * 4 + 2: return launch_solo_gemm_form<GEMM_NVFP4, EPI_F32, 2>(p, grid, smem, stream);
        case EPI_BF16 * 4 + 1: return launch_solo_gemm_form<GEMM_NVFP4, EPI_BF16, 1>(p, grid, smem, stream);
        case EPI_BF16 * 4 + 2: return launch_solo_gemm_form<GEMM_NVFP4, EPI_BF16, 2>(p, grid, smem, stream);
        case EPI_FP4 * 4 + 1: return launch_solo_gemm_form<GEMM_NVFP4, EPI_FP4, 1>(p, grid, smem, stream);
        case EPI_FP4 * 4 + 2: return launch_solo_gemm_form<GEMM_NVFP4, EPI_FP4, 2>(p, grid, smem, stream);
        case EPI_GEGLU_FP4 * 4 + 1: return launch_solo_gemm_form<GEMM_NVFP4, EPI_GEGLU_FP4, 1>(p, grid, smem, stream);
        case EPI_GEGLU_FP4 * 4 + 2: return launch_solo_gemm_form<GEMM_NVFP4, EPI_GEGLU_FP4, 2>(p, grid, smem, stream);
        default: return cudaErrorNotSupported;
    }
}
}  // namespace pi0


