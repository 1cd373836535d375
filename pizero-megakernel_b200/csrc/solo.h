// Kernels of their own for operators that are launched by themselves.
//
// A program of many stages runs in the persistent kernel (vm_kernel.cuh).  One operator alone pays for what that kernel is built for -
// descriptors fetched from memory, one CTA of 224 KiB per SM, eight warps that change roles, tiles of one SM - and gains nothing from
// it, so the operators that a user launches one at a time have kernels here whose arguments arrive with the launch.  They compute what the
// stage of a program computes; launch_solo decides which operators go this way, and the others run as a program of one stage as before.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "vm_types.h"

namespace pi0 {

// What every kernel needs beside its operands: where to report a wait that ran out, and how long it may take.
struct SoloGuard {
    VmStatus* status;
    unsigned long long budget_ns;
    unsigned int* counters;      // finished tiles per 128-row band, as the stage of a program leaves them
    int early;                   // let the next launch of the stream prepare while this one runs
};

struct SoloNorm {
    NormParams n;
    SoloGuard guard;
};

struct alignas(64) SoloGemm {
    CUtensorMap map_a, map_b;    // rows of A as [chunk][row][128 bytes]; of B as [block][chunk][row][128 bytes] (one block when row-major)
    CUtensorMap map_sfa, map_sfb;    // scale atoms (pairs of CTAs only): of A [atom][512 bytes], of B [row tile][K group][512 bytes]
    GemmParams g;                // operands, epilogue; bn, idesc and the ring below replace its tile geometry
    SoloGuard guard;
    int items;                   // tiles
    int m_tiles, n_tiles;        // tiles of tile_rows (x 2 in pairs) x bn
    int bn, tile_rows;
    int splits;                  // K splits: pairs of a cluster that share a tile
    int chunks, slots;           // 128-byte chunks of K and slots of kc chunks
    int stages, stride, off_b, off_sfa, off_sfb;     // operand ring
    int a_rows;                  // rows of A per copy
    int b_rows, b_boxes;         // rows of B per copy, copies per chunk
    int b_block;                 // rows of one block of B
    int sfb_atoms;               // scale atoms of B per K group of a tile
    int sfb_per_tile;            // scale atoms of B start at the tile's ordinal (32-wide tiles) instead of its first row
    int acc_bufs, acc_stride;    // accumulators in tensor memory, columns from one to the next
    int sf_col, sf_mask, tmem_cols;  // first scale column, slots whose scales alternate (mask), columns allocated
};

struct alignas(64) SoloAttn {
    CUtensorMap map_q, map_k, map_v;     // BF16 [image][row][columns] with boxes of 64 columns
    CUtensorMap map_out;         // rows of the output, or of the partial rows
    SoloGuard guard;
    void* out;                   // BF16 [rows, 256]
    uint16_t* partial_o;         // BF16 bits [row tile][split][128][256]
    float* partial_ml;           // FP32 [row tile][split][128][2]
    unsigned int* tickets;       // program counters: 64-column pieces (4 a CTA) whose partial rows are out, per row tile, over all launches ...
    unsigned int target;         // ... and how many that will be after this one
    int rows, heads;             // rows of Q that tiles are cut from: queries x heads, or the queries of an image (heads apart)
    int head_dim, group, query_tiles;    // heads apart: logical columns of a head, query heads per KV head, tiles per image
    int keys, splits, per, cols; // keys of a split, score columns computed for them (a multiple of 16, at most 256)
    int items;                   // row tiles x splits
    int off_k, off_v, ctl_offset;    // shared memory: Q and P at 0, K, V
    int prefix;
    float scale;
};
struct SoloAttnPlan {
    SoloAttn args;
    int grid, row_tiles;
    size_t smem;
};
cudaError_t plan_solo_attention(const AttnParams& a, int workers, int sms, SoloAttnPlan* plan);
cudaError_t launch_solo_attention(const SoloAttn& p, int grid, size_t smem, cudaStream_t stream);

// What a GEMM handle asks for; tile geometry and ring of `g` are the persistent kernel's and are not read.
struct SoloGemmRequest {
    const GemmParams* g;
    const void *a, *b;
    int m, n, k, operands, workers;
};
// How it is launched.
struct SoloGemmPlan {
    SoloGemm args;
    int cg, grid;
    size_t smem;
};
// cudaErrorNotSupported: this form runs as a program of one stage.
cudaError_t plan_solo_gemm(const SoloGemmRequest& r, SoloGemmPlan* plan);

cudaError_t launch_solo_norm(const SoloNorm& p, int grid, int groups, cudaStream_t stream);
// Both return cudaErrorNotSupported for a combination that has no kernel.
cudaError_t launch_solo_gemm_nvfp4(const SoloGemm& p, int cg, int grid, size_t smem, cudaStream_t stream);
cudaError_t launch_solo_gemm_dense(const SoloGemm& p, int cg, int grid, size_t smem, cudaStream_t stream);

// Draining warps: as many as the registers of the epilogue allow.  One 32-column piece is a serial chain of some 1,800 cycles, whose latency only
// other warps can fill (gate/up of 768 rows 31 us with eight, 29 with sixteen).
__host__ __device__ constexpr int solo_drain_warps(int operands, int epi) {
    return epi == EPI_GEGLU_FP4 || (epi == EPI_F32 && operands == GEMM_NVFP4) ? 16 : epi == EPI_F32 ? 8 : 12;
}
// Clusters of `ctas` CTAs with all of an SM's shared memory that are resident at once (B200: 74 of 2, 33 of 4, 22 of 6, 15 of 8).
int solo_gemm_clusters(int ctas);

constexpr int kSoloChunks1 = 2, kSoloChunks2 = 1;    // 128-byte chunks of K per slot: tiles of one CTA, of a pair
constexpr int kSoloMaxSlots = 8;
constexpr int kSoloCtlBytes = 1024;
constexpr int kSoloMaxSmem = 227 * 1024;
constexpr int kSoloAttnCtl = 5120;                   // barriers, exchange of the softmax
constexpr int kSoloDataBytes = 225 * 1024;

}  // namespace pi0
