// Tile geometry, operand ring and tensor maps of the GEMM that is launched by itself.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <numeric>

#include "solo.h"

namespace pi0 {
namespace {

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encoder() {
    static const EncodeTiled fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        const bool ok = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess;
        return ok ? reinterpret_cast<EncodeTiled>(p) : nullptr;
    }();
    return fn;
}
cudaError_t encode(CUtensorMap* map, const void* base, CUtensorMapDataType type, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box,
                   CUtensorMapSwizzle swizzle) {
    const EncodeTiled fn = encoder();
    if (!fn) return cudaErrorNotSupported;
    const cuuint32_t ones[4] = {1u, 1u, 1u, 1u};
    const CUresult r = fn(map, type, rank, const_cast<void*>(base), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

struct Shape {
    int cg, bn, tile_rows, splits;
};

// Estimated microseconds of a launch in this shape: the longest of what one SM takes in, what all of them draw from L2 together, MMAs and drains,
// and the last drain.  Rates and cycles per MMA group as measured on single shapes; on 70 projections of 1 to 820 rows (NVFP4, BF16 and FP8, all
// widths of the model and odd ones) in up to ten shapes each, 3.6 - 60 us, the choice is 0.1 % slower than the fastest shape on average, 7 % at
// most.
double estimate(const SoloGemmRequest& r, const Shape& s, int chunks, int a_rows) {
    const GemmParams& g = *r.g;
    const bool scaled = r.operands == GEMM_NVFP4;
    const int row_tiles = ((g.rows + s.tile_rows - 1) / s.tile_rows + s.cg - 1) / s.cg, col_tiles = (g.cols + s.bn - 1) / s.bn;
    const int ctas = s.cg * s.splits, items = row_tiles * col_tiles, units = std::min(r.workers / ctas, solo_gemm_clusters(ctas)), rounds = (items + units - 1) / units;
    const double k_chunks = static_cast<double>(chunks) / s.splits;
    const double rows = a_rows + static_cast<double>(s.bn) / s.cg + (scaled ? (128.0 + (s.bn + 127) / 128 * 128) / 8 : 0.0);
    const double bytes = rows * 128.0 * k_chunks;                                            // of one CTA and tile
    const double copy = std::max(rounds * bytes / 150e3, items * ctas * bytes / 14.6e6);
    const double group = scaled ? (s.cg == 1 ? std::max(40.0, 0.8 * s.bn) : 96 + 0.04 * s.bn) : s.cg == 1 ? 45 + 0.2 * s.bn : std::max(43.0, 0.29 * s.bn);
    const double mma = rounds * k_chunks * 4.0 * group / 1.9e3;
    const int shares = solo_drain_warps(r.operands, g.epilogue) / 4;
    const double drain = (s.bn / 32 + shares - 1) / shares * (g.epilogue == EPI_F32 ? 0.44 : 0.55);
    return 3.4 + (s.cg == 2 ? 2.0 : 0.0) + (s.splits > 1 ? 1.5 : 0.0) + 0.1 * rounds + std::max({copy, mma, rounds > 1 ? rounds * drain : 0.0}) + drain;
}

}  // namespace

cudaError_t plan_solo_gemm(const SoloGemmRequest& r, SoloGemmPlan* plan) {
    const GemmParams& g = *r.g;
    const bool scaled = r.operands == GEMM_NVFP4;
    const bool plain = g.epilogue == EPI_F32 || g.epilogue == EPI_BF16 || (scaled && (g.epilogue == EPI_FP4 || g.epilogue == EPI_GEGLU_FP4));
    if (!plain || g.row_factor || g.row_sumsq || g.round_before_residual || g.gelu_cols > 0 || g.pad_from > 0 || g.col_center || g.cols != r.n || g.block_n > 128)
        return cudaErrorNotSupported;
    if (scaled && g.epilogue == EPI_F32 && (g.bias || g.residual)) return cudaErrorNotSupported;
    // At most 64 rows to BF16 on at most 32 tiles of 64 columns: the MMAs of a long K are all there is, and over 16384 and more the persistent kernel issues
    // them as fast and has its first operands earlier.  Stage and own kernel (us): x 2048 x 16384 1 row 14.8 and 15.4, 64 rows 15.4 and 15.4; 73
    // rows, whose tiles copy more of A, 17.3 and 15.5; x 4096 x 16384, where twice the CTAs share L2, 16.6 and 16.0; x 2048 x 12544 51 rows 13.2 and 12.9;
    // x 2048 x 32768 24.4 and 26.6.  (51 rows to FP32 15.2 and 14.9.)
    if (scaled && g.epilogue == EPI_BF16 && g.rows <= 64 && r.k >= 16384 && g.block_n == 64 && g.cols <= 32 * 64 && g.cols <= r.workers * 64) return cudaErrorNotSupported;
    const size_t row_bytes = scaled ? static_cast<size_t>(r.k) / 2 : r.operands == GEMM_BF16 ? static_cast<size_t>(r.k) * 2 : static_cast<size_t>(r.k);
    const int chunks = static_cast<int>((row_bytes + 127) / 128), k_groups = static_cast<int>(row_bytes / 32);
    const int few = std::min(128, std::max(scaled ? 32 : 64, (g.rows + 7) / 8 * 8));          // rows copied when there is one row band
    const bool own_atoms = scaled && g.block_n == 32;                                         // scales in the layout of 32-wide tiles

    Shape best{};
    double least = 0;
    for (const int cg : {1, 2}) {
        if (cg == 2 && (r.workers < 2 || r.m == 128 || own_atoms)) continue;
        for (const int bn : {32, 64, 128, 192, 256}) {
            if (own_atoms ? bn != 32 : scaled && bn < 64) continue;
            if (bn > (cg == 1 ? 128 : scaled ? 192 : 256) || (cg == 2 && bn < 64)) continue;
            for (const int tile_rows : {128, 64}) {
                if (tile_rows == 64 && (scaled || cg == 2 || r.m == 128)) continue;
                for (const int splits : {1, 2, 3, 4}) {
                    if (splits > 1 && (scaled || cg == 1 || chunks < 32 * splits)) continue;
                    if (std::min(r.workers / (cg * splits), solo_gemm_clusters(cg * splits)) < 1) continue;
                    const int tiles = ((g.rows + 255) / 256) * ((g.cols + bn - 1) / bn);
                    if (splits > 1 && tiles > std::min(r.workers / (2 * splits), solo_gemm_clusters(2 * splits))) continue;      // (one tile per cluster)
                    const Shape s{cg, bn, tile_rows, splits};
                    const double t = estimate(r, s, chunks, r.m == 128 ? few : tile_rows);
                    if (least == 0 || t < least) { best = s; least = t; }
                }
            }
        }
    }
    if (least == 0) return cudaErrorNotSupported;

    memset(plan, 0, sizeof(*plan));
    SoloGemm& p = plan->args;
    p.g = g;
    p.g.k_groups = k_groups;
    p.g.operands = r.operands;
    const int kc = best.cg == 2 ? kSoloChunks2 : kSoloChunks1;
    p.bn = best.bn;
    p.tile_rows = best.tile_rows;
    p.splits = best.splits;
    p.m_tiles = ((g.rows + best.tile_rows - 1) / best.tile_rows + best.cg - 1) / best.cg;
    p.n_tiles = (g.cols + best.bn - 1) / best.bn;
    p.items = p.m_tiles * p.n_tiles;
    p.chunks = chunks;
    p.slots = (chunks + kc - 1) / kc;
    p.a_rows = r.m == 128 ? few : best.tile_rows;
    p.b_block = g.b_tiled ? g.block_n : r.n;
    const int b_rows = best.bn / best.cg;
    p.b_rows = g.b_tiled ? std::gcd(g.block_n, b_rows) : b_rows;
    p.b_boxes = b_rows / p.b_rows;
    p.sfb_per_tile = own_atoms ? 1 : 0;
    p.sfb_atoms = !scaled ? 0 : best.bn > 128 ? 2 : 1;
    const int sf_bytes = scaled ? kc * 4 * 512 : 0;
    p.off_b = kc * 128 * p.a_rows;
    p.off_sfa = p.off_b + kc * 128 * b_rows;
    p.off_sfb = p.off_sfa + sf_bytes;
    p.stride = p.off_sfb + sf_bytes * p.sfb_atoms;
    // (the MMA reads 128 rows of A, of which a_rows were copied: the rest has to lie inside the slot)
    p.stride = std::max(p.stride, ((kc - 1) * 128 * p.a_rows + 128 * 128 + 1023) / 1024 * 1024);
    const int units = std::min({r.workers / (best.cg * best.splits), solo_gemm_clusters(best.cg * best.splits), p.items}), rounds = (p.items + units - 1) / units;
    plan->cg = best.cg;
    plan->grid = units * best.cg * best.splits;
    p.stages = std::min({kSoloMaxSlots, kSoloDataBytes / p.stride, rounds * ((p.slots + best.splits - 1) / best.splits)});
    // (a split of K: the others' sums for this pair's share of the columns take the place of the ring.  16 KiB per 32-column piece and other pair, at
    // most 96 KiB - 256 columns in 3 or 4 parts - where the ring of 32 slots and more per part has at least 160)
    plan->smem = kSoloCtlBytes + static_cast<size_t>(p.stages) * p.stride + 1024;
    // tensor memory: one or two accumulators, behind them the scales of two or four slots
    p.acc_bufs = rounds > 1 ? 2 : 1;
    p.acc_stride = best.bn;
    const int sf_slot = scaled ? 4 * kc * (4 + 4 * p.sfb_atoms) : 0, sf_bufs = p.sfb_atoms == 2 ? 2 : 4;
    p.sf_col = (p.acc_bufs * p.acc_stride + 3) / 4 * 4;
    p.sf_mask = sf_bufs - 1;
    int cols = 32;
    while (cols < p.sf_col + sf_slot * sf_bufs) cols *= 2;
    if (cols > 512) return cudaErrorNotSupported;
    p.tmem_cols = cols;
    const uint32_t fmt = r.operands == GEMM_FP8 ? 0u : 1u, acc_f32 = scaled ? 0u : 1u << 4;
    p.g.idesc = acc_f32 | (fmt << 7) | (fmt << 10) | (static_cast<uint32_t>(best.bn >> 3) << 17) | (static_cast<uint32_t>((128 * best.cg) >> 4) << 24);

    const cuuint64_t a_dims[3] = {128u, static_cast<cuuint64_t>(r.m), static_cast<cuuint64_t>(chunks)}, a_strides[2] = {row_bytes, 128u};
    const cuuint32_t a_box[3] = {128u, static_cast<cuuint32_t>(p.a_rows), static_cast<cuuint32_t>(kc)};
    cudaError_t e = encode(&p.map_a, r.a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, a_dims, a_strides, a_box, CU_TENSOR_MAP_SWIZZLE_128B);
    const cuuint64_t block = static_cast<cuuint64_t>(p.b_block);
    const cuuint64_t b_dims[4] = {128u, block, static_cast<cuuint64_t>(chunks), static_cast<cuuint64_t>(r.n) / block};
    const cuuint64_t b_strides[3] = {g.b_tiled ? 128u : row_bytes, g.b_tiled ? block * 128u : 128u, row_bytes * block};
    const cuuint32_t b_box[4] = {128u, static_cast<cuuint32_t>(p.b_rows), static_cast<cuuint32_t>(p.b_boxes == 1 ? kc : 1), 1u};
    if (e == cudaSuccess) e = encode(&p.map_b, r.b, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, b_dims, b_strides, b_box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (e == cudaSuccess && scaled && best.cg == 2) {
        const cuuint64_t strides[2] = {512u, static_cast<cuuint64_t>(k_groups) * 512u};
        const cuuint32_t box[3] = {128u, static_cast<cuuint32_t>(4 * kc), static_cast<cuuint32_t>(p.sfb_atoms)};
        const cuuint64_t a_atoms[2] = {128u, static_cast<cuuint64_t>(r.m / 128) * k_groups};
        const cuuint64_t b_atoms[3] = {128u, static_cast<cuuint64_t>(k_groups), static_cast<cuuint64_t>(r.n / 128)};
        e = encode(&p.map_sfa, g.sfa, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, a_atoms, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
        if (e == cudaSuccess) e = encode(&p.map_sfb, g.sfb, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, b_atoms, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
    }
    return e;
}

cudaError_t plan_solo_attention(const AttnParams& a, int workers, int sms, SoloAttnPlan* plan) {
    const bool shared_kv = a.batches == 1 && a.kv_heads == 1 && a.head_dim == 256 && a.hd_pad == 256 && a.ldq == a.heads * 256 && a.ldo == a.heads * 256;
    const bool apart_heads = a.hd_pad == 128 && a.splits == 1;
    if (!a.tc || a.mask || a.out_fp4 || !a.out || !(shared_kv || apart_heads)) return cudaErrorNotSupported;
    memset(plan, 0, sizeof(*plan));
    SoloAttn& p = plan->args;
    p.rows = shared_kv ? a.nq * a.heads : a.nq;
    p.head_dim = a.head_dim;
    p.group = a.heads / a.kv_heads;
    p.query_tiles = (a.nq + 127) / 128;
    const int pieces = a.hd_pad / 64;
    const int row_tiles = (p.rows + 127) / 128;
    // The ranges of keys are the handle's: each is a maximum that probabilities are rounded against and a partial row that is rounded, so other
    // ranges are other results, and fewer are less exact (784 rows in 3 ranges instead of 4: one round of SMs and 16.1 us, not two and 23.7, but
    // 2.746e-3 from 64 bits and not 2.724e-3; 10 queries over 487 keys in 11 ranges instead of 13: 2.646e-3 and not 2.574e-3).
    p.splits = a.splits;
    p.per = (a.nk + a.splits - 1) / a.splits;
    p.cols = (p.per + 15) / 16 * 16;                                                          // (at most 256, or the tiles would not be tcgen05 ones)
    p.keys = a.nk;
    p.heads = a.heads;
    p.items = shared_kv ? row_tiles * p.splits : a.batches * p.query_tiles * a.heads;
    p.prefix = a.prefix;
    p.scale = a.scale;
    p.out = a.out;
    p.partial_o = a.partial_o;
    p.partial_ml = a.partial_ml;
    plan->row_tiles = row_tiles;
    plan->grid = std::min(p.items, std::min(workers, sms));
    const int first = std::max(pieces, (p.cols + 63) / 64) * 16384, kv = pieces * p.cols * 128;     // Q, later P and the output; K or V
    p.off_k = first;
    const bool apart = first + 2 * kv + kSoloAttnCtl + 1024 <= kSoloMaxSmem;
    p.off_v = apart ? first + kv : first;
    p.ctl_offset = p.off_v + kv;
    plan->smem = p.ctl_offset + kSoloAttnCtl + 1024;
    if (plan->smem > static_cast<size_t>(kSoloMaxSmem)) return cudaErrorNotSupported;
    const cuuint64_t images = static_cast<cuuint64_t>(a.batches), out_bytes = static_cast<cuuint64_t>(a.ldo) * 2u;
    const cuuint64_t q_width = shared_kv ? 256u : static_cast<cuuint64_t>(a.heads) * 128u, q_ld = shared_kv ? 512u : static_cast<cuuint64_t>(a.ldq) * 2u;
    const cuuint64_t q_dims[3] = {q_width, static_cast<cuuint64_t>(p.rows), images}, q_strides[2] = {q_ld, q_ld * static_cast<cuuint64_t>(shared_kv ? p.rows : a.q_batch_rows)};
    const cuuint32_t q_box[3] = {64u, 128u, 1u};
    const cuuint64_t kv_ld = static_cast<cuuint64_t>(a.ldkv) * 2u;
    const cuuint64_t kv_dims[3] = {static_cast<cuuint64_t>(a.kv_heads * a.hd_pad), static_cast<cuuint64_t>(a.kv_batch_rows), images}, kv_strides[2] = {kv_ld, kv_ld * static_cast<cuuint64_t>(a.kv_batch_rows)};
    const cuuint32_t kv_box[3] = {64u, static_cast<cuuint32_t>(p.cols), 1u};
    cudaError_t e = encode(&p.map_q, a.q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, q_dims, q_strides, q_box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (e == cudaSuccess) e = encode(&p.map_k, a.k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, kv_dims, kv_strides, kv_box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (e == cudaSuccess) e = encode(&p.map_v, a.v, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, kv_dims, kv_strides, kv_box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (e != cudaSuccess) return e;
    if (shared_kv) {
        const cuuint64_t dims[2] = {256u, static_cast<cuuint64_t>(p.splits > 1 ? p.items * 128 : p.rows)}, strides[1] = {512u};
        return encode(&p.map_out, p.splits > 1 ? static_cast<const void*>(a.partial_o) : a.out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dims, strides, q_box, CU_TENSOR_MAP_SWIZZLE_128B);
    }
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(a.heads * a.head_dim), static_cast<cuuint64_t>(a.nq), images};
    const cuuint64_t strides[2] = {out_bytes, out_bytes * static_cast<cuuint64_t>(a.q_batch_rows)};
    const cuuint32_t box[3] = {static_cast<cuuint32_t>(a.head_dim), 128u, 1u};
    return encode(&p.map_out, a.out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
}

}  // namespace pi0
