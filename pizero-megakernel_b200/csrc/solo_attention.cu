// Attention launched by itself: softmax(scale * Q K^T + suffix mask) V.
//
// PIECES = 4: query heads that share one KV head of 256 (Gemma).  With one KV head the rows (query, head) all read the same keys, and they lie one behind another in memory: Q is one matrix of
// queries x heads rows of 256, cut into tiles of 128 rows whatever the number of queries is.  A work item is one such tile against one range of
// keys (KV split); 784 queries of 8 heads in 4 ranges are 196 items, where tiles per head (7 x 8, the last of each with 16 rows) are 224.
// PIECES = 2: heads of at most 128, stored 128 apart (SigLIP), with at most 256 keys: an item is 128 queries of one head of one image, no splits.
//
// Three images of 256 queries, 16 heads: 7.4 us (as a program of one stage 10.8), one image of 200 6.7 (9.7).
//
//   warp 0       copies: Q and K in pieces of 64 columns, V likewise (behind K, or in K's place once the scores are complete)
//   warp 1       tensor memory; S = Q K^T piece by piece as they land, O = P V
//   warps 2-17   four threads per row: row maximum, exponentials, P in BF16 over Q, then a quarter of O's columns each
//
// What bounds it: a chain of copies, scores, softmax, MMAs, one trip to L2 with the partial rows and one back (51 queries over 819 keys, 13 splits:
// scores complete 1.6 us after the release, O 3.2, partial rows out and counted 5.9, merged 8.7, next launch released 10.0; the tiles per
// head of a program's stage 12.2); with 196 keys a tile 25,000 exponentials per SM and item besides, and where there are more items than SMs
// the second one's copies wait for the first one's output (784 queries: 23.7 us, tiles per head 29.5; 623 in 3 ranges, one round, 13.4 and 17.1).  The
// splits of a tile as a cluster that exchanges its rows through shared memory, by stores or by copies, were no faster (10.8).
//
// S takes up to 256 columns of tensor memory and O those from 256 on.  Ranges of keys, those that the operator was given, meet as
// un-normalised BF16 rows with their maximum and sum (as in op_attention_tc.cuh): when all of a tile's ranges have arrived, each of their
// CTAs merges a share of the rows.
#include "op_attention.cuh"
#include "solo.h"
#include "solo_common.cuh"

namespace pi0 {

constexpr int kSoloAttnThreads = 576;

struct SoloAttnCtl {
    uint64_t k[4], s, p, v[4], o, free;
    uint32_t tmem;
    int abort;
    float xm[4][128], xl[4][128];    // row maxima and sums of the four threads of a row
};

static_assert(sizeof(SoloAttnCtl) <= kSoloAttnCtl, "control block of the attention kernel");

// Weights of a row's splits: lane s has the maximum and sum of split s (and s + 32); afterwards its weight over the row's sum.
__device__ __forceinline__ float2 split_weights(float2 lo, float2 hi) {
    float big = fmaxf(lo.x, hi.x);
#pragma unroll
    for (int o = 16; o; o >>= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
    const float ref = big == -INFINITY ? 0.f : big;
    const float w_lo = exp2_fast(lo.x - ref), w_hi = exp2_fast(hi.x - ref);                  // 0 for an absent or fully masked split
    float denom = w_lo * lo.y + w_hi * hi.y;
#pragma unroll
    for (int o = 16; o; o >>= 1) denom += __shfl_xor_sync(0xffffffffu, denom, o);
    const float inv = denom > 0.f ? 1.f / denom : 0.f;
    return make_float2(w_lo * inv, w_hi * inv);
}
__device__ __forceinline__ void add_weighted(float2 (&acc)[4], float w, uint4 x) {
    const uint32_t u[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int e = 0; e < 4; e++) acc[e] = fma2(make_float2(w, w), __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[e])), acc[e]);
}
__device__ __forceinline__ uint4 pack_row(const float2 (&acc)[4]) {
    return make_uint4(pack2_bf16(acc[0].x, acc[0].y), pack2_bf16(acc[1].x, acc[1].y), pack2_bf16(acc[2].x, acc[2].y), pack2_bf16(acc[3].x, acc[3].y));
}

// Where a work item begins: its rows of Q, its keys, the columns of its heads.
struct AttnItem {
    int row0, key0, q_column, kv_column, batch, head;
};
template <int PIECES>
__device__ __forceinline__ AttnItem attn_item(const SoloAttn& p, int item) {
    if constexpr (PIECES == 4) {
        const int row_tile = item / p.splits;
        return {row_tile * 128, (item - row_tile * p.splits) * p.per, 0, 0, 0, 0};
    } else {
        const int tile = item / p.heads, head = item - tile * p.heads, batch = tile / p.query_tiles;
        return {(tile - batch * p.query_tiles) * 128, 0, head * 128, head / p.group * 128, batch, head};
    }
}

// Counter of a finished item: the 128-query band in which its row tile begins, or its tile of an image.
template <int PIECES>
__device__ __forceinline__ unsigned int attn_band(const SoloAttn& p, int item) {
    return PIECES == 4 ? static_cast<unsigned>(item / p.splits) / static_cast<unsigned>(p.heads) : static_cast<unsigned>(item / p.heads);
}

template <int PIECES>
__global__ void __launch_bounds__(kSoloAttnThreads, 1) pi0_attention_kernel(const __grid_constant__ SoloAttn p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* data = base;
    SoloAttnCtl* ctl = reinterpret_cast<SoloAttnCtl*>(base + p.ctl_offset);
    const int warp = threadIdx.x >> 5, lane = lane_id();
    if (threadIdx.x == 0) {
        for (int c = 0; c < PIECES; c++) {
            mbar_init(&ctl->k[c], 1);
            mbar_init(&ctl->v[c], 1);
        }
        mbar_init(&ctl->s, 1);
        mbar_init(&ctl->o, 1);
        mbar_init(&ctl->p, 16);
        mbar_init(&ctl->free, PIECES == 4 ? 4 : 1);
        ctl->abort = 0;
        mbar_fence_init();
        prefetch_tmap(&p.map_q);
        prefetch_tmap(&p.map_k);
        prefetch_tmap(&p.map_v);
        prefetch_tmap(&p.map_out);
    }
    if (warp == 1) tmem_alloc_cg<1>(&ctl->tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctl->tmem;
    const SoloWait w{p.guard.status, p.guard.budget_ns, &ctl->abort};
    const int items = p.items, splits = p.splits, per = p.per, cols = p.cols;
    const uint32_t slab = static_cast<uint32_t>(cols) * 128u;              // one 64-column piece of K or V
    uint8_t *sk = data + p.off_k, *sv = data + p.off_v;
    const bool v_apart = p.off_v != p.off_k;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t n = 0;
            bool alive = true;
            grid_dependency_wait();
            for (int item = blockIdx.x; alive && item < items; item += gridDim.x, ++n) {
                const AttnItem at = attn_item<PIECES>(p, item);
                if (n > 0 && !solo_wait(w, &ctl->free, (n - 1) & 1u)) break;
#pragma unroll
                for (int c = 0; c < PIECES; ++c) {
                    mbar_expect_tx(&ctl->k[c], 16384u + slab);
                    tma_load_3d(data + c * 16384, &p.map_q, &ctl->k[c], at.q_column + c * 64, at.row0, at.batch);
                    tma_load_3d(sk + static_cast<uint32_t>(c) * slab, &p.map_k, &ctl->k[c], at.kv_column + c * 64, at.key0, at.batch);
                }
                if (!v_apart && !solo_wait(w, &ctl->s, n & 1u)) break;
#pragma unroll
                for (int c = 0; c < PIECES; ++c) {
                    mbar_expect_tx(&ctl->v[c], slab);
                    tma_load_3d(sv + static_cast<uint32_t>(c) * slab, &p.map_v, &ctl->v[c], at.kv_column + c * 64, at.key0, at.batch);
                }
            }
        }
    } else if (warp == 1) {
        const uint32_t tmem_u = uniform_u32(tmem), q16 = uniform_u32((smem_u32(data) & 0x3FFFFu) >> 4), k16 = uniform_u32((smem_u32(sk) & 0x3FFFFu) >> 4),
                       v16 = uniform_u32((smem_u32(sv) & 0x3FFFFu) >> 4), slab16 = uniform_u32(slab >> 4);
        if (elect_one()) {
            constexpr uint64_t kKMajor = (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
            constexpr uint32_t kBf16 = (1u << 4) | (1u << 7) | (1u << 10) | (8u << 24);
            const uint32_t idesc_s = kBf16 | ((static_cast<uint32_t>(cols) >> 3) << 17), idesc_o = kBf16 | (1u << 16) | ((PIECES * 64u >> 3) << 17);
            const int steps = cols >> 4;
            uint32_t n = 0;
            bool alive = true;
            for (int item = blockIdx.x; alive && item < items; item += gridDim.x, ++n) {
#pragma unroll 1
                for (uint32_t c = 0; alive && c < PIECES; ++c) {
                    if (!solo_wait(w, &ctl->k[c], n & 1u)) { alive = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i) {
                        tc_mma_f16(tmem_u, kKMajor | static_cast<uint64_t>(q16 + c * 1024u + 2u * i), kKMajor | static_cast<uint64_t>(k16 + c * slab16 + 2u * i), idesc_s,
                                   (c | i) != 0u ? 1u : 0u);
                    }
                }
                if (!alive) break;
                tc_commit(&ctl->s);
                if (!solo_wait(w, &ctl->p, n & 1u)) break;
                tc_fence_after();
                for (uint32_t c = 0; alive && c < PIECES; ++c) alive = solo_wait(w, &ctl->v[c], n & 1u);
                if (!alive) break;
                tc_fence_after();
                // B = V with the columns of the head contiguous: pieces of 64 columns one slab apart, one 128-byte row per key, groups of 8 keys 1 KiB apart
                const uint64_t v_major = (static_cast<uint64_t>(slab16) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
#pragma unroll 4
                for (uint32_t j = 0; j < static_cast<uint32_t>(steps); ++j)
                    tc_mma_f16(tmem_u + 256u, kKMajor | static_cast<uint64_t>(q16 + (j >> 2) * 1024u + 2u * (j & 3u)), v_major | static_cast<uint64_t>(v16 + j * 128u), idesc_o,
                               j != 0 ? 1u : 0u);
                tc_commit(&ctl->o);
            }
        }
    } else {
        // Every warp goes through the same barriers whatever its waits say: one that ran out only leaves the work undone.
        const int quarter = warp & 3, share = (warp - 2) >> 2;
        const int row = quarter * 32 + lane;
        const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
        const float sl2 = p.scale * 1.4426950408889634f;
        const int groups = cols >> 4, g0 = groups * share >> 2, g1 = groups * (share + 1) >> 2;
        uint32_t n = 0;
        bool alive = true;
        grid_dependency_wait();
        if (p.guard.early) grid_launch_dependents();
        for (int item = blockIdx.x; item < items; item += gridDim.x, ++n) {
            const AttnItem at = attn_item<PIECES>(p, item);
            const int row_tile = item / splits, k_begin = at.key0;
            const int keys = max(min(p.keys - k_begin, per), 0);
            const int tile_row = at.row0 + row, warp_rows = p.rows - (tile_row - lane);
            const int visible = p.prefix >= 0 && tile_row < (PIECES == 4 ? p.heads : 1) ? min(keys, p.prefix + 1 - k_begin) : keys;     // (query 0)
            alive = alive && solo_wait_warp(w, &ctl->s, n & 1u);
            tc_fence_after();
            uint32_t raw[16];
            auto scores = [&](int j) {                       // 16 scores of this row, hidden keys at -infinity
                tmem_ld16(lane_addr + j * 16, raw);
                tmem_ld_wait();
                const int open = visible - j * 16;
                if (__any_sync(0xffffffffu, open < 16)) {
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        if (i >= open) raw[i] = 0xff800000u;
                }
            };
            float m_part = -INFINITY;
            if (alive && warp_rows > 0) {
#pragma unroll 1
                for (int j = g0; j < g1; ++j) {
                    scores(j);
                    float m4[4] = {m_part, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                    for (int i = 0; i < 16; i += 8)
#pragma unroll
                        for (int e = 0; e < 4; e++) m4[e] = max3(m4[e], __uint_as_float(raw[i + 2 * e]), __uint_as_float(raw[i + 2 * e + 1]));
                    m_part = fmaxf(max3(m4[0], m4[1], m4[2]), m4[3]);
                }
            }
            ctl->xm[share][row] = m_part;
            named_barrier(1 + quarter, 128);
            const float m_raw = fmaxf(max3(ctl->xm[0][row], ctl->xm[1][row], ctl->xm[2][row]), ctl->xm[3][row]);
            const float m_use = m_raw == -INFINITY ? 0.f : m_raw * sl2;
            float2 l_part = make_float2(0.f, 0.f);
            if (alive && warp_rows > 0) {
#pragma unroll 1
                for (int j = g0; j < g1; ++j) {
                    scores(j);
                    uint32_t packed[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const float2 x = fma2(make_float2(__uint_as_float(raw[2 * i]), __uint_as_float(raw[2 * i + 1])), make_float2(sl2, sl2), make_float2(-m_use, -m_use));
                        const float2 e = make_float2(exp2_fast(x.x), exp2_fast(x.y));
                        l_part = add2(l_part, e);
                        packed[i] = pack2_bf16(e.x, e.y);
                    }
                    uint8_t* dst = data + (j >> 2) * 16384 + row * 128;
#pragma unroll
                    for (int u = 0; u < 2; u++)
                        *reinterpret_cast<uint4*>(dst + (((j & 3) * 2 + u) ^ (row & 7)) * 16) = make_uint4(packed[4 * u], packed[4 * u + 1], packed[4 * u + 2], packed[4 * u + 3]);
                }
            }
            ctl->xl[share][row] = l_part.x + l_part.y;
            tc_fence_before();
            fence_proxy_async_smem();                        // P (generic stores) before the tensor core's reads
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctl->p);
            named_barrier(1 + quarter, 128);
            const float l_sum = (ctl->xl[0][row] + ctl->xl[1][row]) + (ctl->xl[2][row] + ctl->xl[3][row]);
            const float inv = l_sum > 0.f ? 1.f / l_sum : 0.f;
            const float2 ml = make_float2(m_raw == -INFINITY ? -INFINITY : m_use, l_sum);
            if (PIECES == 4 && splits > 1 && share == 3 && warp_rows > 0) {
                reinterpret_cast<float2*>(p.partial_ml)[static_cast<size_t>(item) * 128 + row] = ml;
                __threadfence();                             // (most of a microsecond, which the MMAs of O cover)
            }
            alive = alive && solo_wait_warp(w, &ctl->o, n & 1u);
            tc_fence_after();
            // 64 columns of O as BF16 over P, whose MMAs are done, in the layout of a swizzled copy
            const float f = splits > 1 ? 1.f : inv;
            uint8_t* piece = PIECES == 4 ? data + share * 16384 + row * 128 : data + row * p.head_dim * 2;     // (PIECES = 2: rows of the head's columns)
            if (alive) {
#pragma unroll 1
                for (int j = 0; j < PIECES; ++j) {
                    const int column = share * (PIECES * 16) + j * 16;
                    tmem_ld16(lane_addr + 256u + column, raw);
                    tmem_ld_wait();
                    uint32_t packed[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) packed[i] = pack2_bf16(__uint_as_float(raw[2 * i]) * f, __uint_as_float(raw[2 * i + 1]) * f);
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const uint4 unit = make_uint4(packed[4 * u], packed[4 * u + 1], packed[4 * u + 2], packed[4 * u + 3]);
                        if constexpr (PIECES == 4) *reinterpret_cast<uint4*>(piece + ((j * 2 + u) ^ (row & 7)) * 16) = unit;
                        else if (column + u * 8 < p.head_dim) *reinterpret_cast<uint4*>(piece + (column + u * 8) * 2) = unit;
                    }
                }
            }
            tc_fence_before();
            fence_proxy_async_smem();
            if constexpr (PIECES == 4) {
                named_barrier(6 + share, 128);               // the piece is complete
                if (quarter == 0 && lane == 0) {
                    // rows beyond the last one are left out by the copy engine
                    if (!solo_gave_up(&ctl->abort)) {
                        tma_store_2d(&p.map_out, data + share * 16384, share * 64, splits > 1 ? item * 128 : at.row0);
                        bulk_store_wait();
                        if (splits > 1) red_release_add(p.tickets + row_tile, 1u);
                    }
                    mbar_arrive(&ctl->free);
                }
            } else {
                named_barrier(6, 512);
                if (warp == 2 && lane == 0) {
                    if (!solo_gave_up(&ctl->abort)) {
                        tma_store_3d(&p.map_out, data, at.head * p.head_dim, at.row0, at.batch);
                        bulk_store_wait();
                    }
                    mbar_arrive(&ctl->free);
                }
            }
            named_barrier(5, 512);                           // (xm and xl are free for the next item)
            if (warp == 2 && lane == 0 && !(PIECES == 4 && splits > 1) && !solo_gave_up(&ctl->abort)) atomicAdd(p.guard.counters + attn_band<PIECES>(p, item), 1u);
        }
        if (PIECES == 4 && splits > 1) {
            // A CTA merges a share of the rows of its tiles.  All CTAs of the grid are resident, and none waits before
            // its own partial rows are out.
            for (int item = blockIdx.x; item < items; item += gridDim.x) {
                const int row_tile = item / splits, split = item - row_tile * splits;
                const int rows = min(128, p.rows - row_tile * 128), r0 = rows * split / splits, mine = rows * (split + 1) / splits - r0;
                int ok = 1;
                if (lane == 0 && warp - 2 < mine) {
                    unsigned long long start = 0;
                    for (uint32_t spin = 1; ok && static_cast<int>(ld_acquire(p.tickets + row_tile) - p.target) < 0; ++spin) {
                        __nanosleep(20);
                        if ((spin & 63u) == 0u) {
                            ok = !solo_gave_up(&ctl->abort);
                            const unsigned long long now = global_ns();
                            if (start == 0) start = now;
                            if (now - start > w.budget_ns || ld_relaxed_int(&w.status->abort)) { solo_give_up(w, 0u); ok = 0; }
                        }
                    }
                }
                if (!__shfl_sync(0xffffffffu, ok, 0)) break;
                __syncwarp();                                // (a shuffle orders no memory: lane 0 has acquired for all of them)
                if (warp == 2 && lane == 0 && !solo_gave_up(&ctl->abort)) atomicAdd(p.guard.counters + attn_band<PIECES>(p, item), 1u);
                const float2* ml = reinterpret_cast<const float2*>(p.partial_ml) + static_cast<size_t>(row_tile) * splits * 128 + r0;
                const uint4* po = reinterpret_cast<const uint4*>(p.partial_o) + (static_cast<size_t>(row_tile) * splits * 128 + r0) * 32 + lane;
                uint4* out = reinterpret_cast<uint4*>(p.out) + (static_cast<size_t>(row_tile) * 128 + r0) * 32 + lane;
                const float2 none = make_float2(-INFINITY, 0.f);
                // (twelve partial rows are on their way together: four splits of three rows, or twelve of one)
                const bool several = splits <= 4;
                for (int i0 = warp - 2; i0 < mine; i0 += several ? 48 : 16) {
                    uint4 x[3][4];
                    float2 lo[3], hi = none;
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        const int i = several ? min(i0 + 16 * k, mine - 1) : i0;
#pragma unroll
                        for (int j = 0; j < 4; j++) x[k][j] = __ldcg(po + (static_cast<size_t>(min(several ? j : 4 * k + j, splits - 1)) * 128 + i) * 32);
                        if (several || k == 0) lo[k] = lane < splits ? __ldcg(ml + lane * 128 + i) : none;
                    }
                    if (splits > 32 && lane + 32 < splits) hi = __ldcg(ml + (lane + 32) * 128 + i0);
                    if (several) {
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            if (i0 + 16 * k >= mine) break;
                            const float2 wt = split_weights(lo[k], none);
                            float2 acc[4] = {};
#pragma unroll
                            for (int j = 0; j < 4; j++)
                                if (j < splits) add_weighted(acc, __shfl_sync(0xffffffffu, wt.x, j), x[k][j]);
                            out[static_cast<size_t>(i0 + 16 * k) * 32] = pack_row(acc);
                        }
                    } else {
                        const float2 wt = split_weights(lo[0], hi);
                        float2 acc[4] = {};
#pragma unroll
                        for (int s = 0; s < 12; s++)
                            if (s < splits) add_weighted(acc, __shfl_sync(0xffffffffu, wt.x, s), x[s >> 2][s & 3]);
#pragma unroll 1
                        for (int s = 12; s < splits; ++s)
                            add_weighted(acc, __shfl_sync(0xffffffffu, s < 32 ? wt.x : wt.y, s & 31), __ldcg(po + (static_cast<size_t>(s) * 128 + i0) * 32));
                        out[static_cast<size_t>(i0) * 32] = pack_row(acc);
                    }
                }
            }
        }
    }
    __syncwarp();
    if (solo_gave_up(&ctl->abort)) {
        const unsigned long long t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc_cg<1>(tmem, 512);
}

namespace {
template <int PIECES>
cudaError_t launch_form(const SoloAttn& p, int grid, size_t smem, cudaStream_t stream) {
    static bool configured[64] = {};
    const auto kernel = pi0_attention_kernel<PIECES>;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    if (device >= 64 || !configured[device]) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSoloMaxSmem);
        if (e != cudaSuccess) return e;
        if (device < 64) configured[device] = true;
    }
    cudaLaunchAttribute serial{};
    serial.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    serial.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(grid);
    config.blockDim = dim3(kSoloAttnThreads);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &serial;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, p);
}
}  // namespace

cudaError_t launch_solo_attention(const SoloAttn& p, int grid, size_t smem, cudaStream_t stream) {
    return p.head_dim == 256 ? launch_form<4>(p, grid, smem, stream) : launch_form<2>(p, grid, smem, stream);
}

}  // namespace pi0
