// GEMM launched by itself:  out[M,N] = epilogue(alpha * A[M,K] . B[N,K]^T), the arithmetic of op_gemm.cuh in a kernel of its own.
//
//   CG = 1: a tile of 128 (or 64) x bn belongs to one CTA.
//   CG = 2: a tile of 256 x bn belongs to a pair of CTAs on neighbouring SMs (cta_group::2).  Each brings 128 rows of A and half of the
//           rows of B, and the tensor cores of both read both halves of B: an SM takes in (128 + bn / 2) rows per 128 x bn of output
//           instead of (128 + bn).
//
//   warp 0      copies of A and its scales         warps 3, 2  copies of B, of its scales
//   warp 1      tensor memory; scale copies and MMAs (in the pair's first CTA)
//   warps 4 ..  drain: warp w the 32 rows of quarter w & 3 and a share of the columns
//
// Pairs of BF16 / FP8 tiles can split K over the pairs of a cluster.
//
// What bounds it: with few rows the chain copies - MMAs - drain (expert q|k|v of 51 rows: 1.2 us to the first operands, 0.8 for its MMAs, 0.7 for
// the drain, 1.3 to the next launch: 4.0 us; as a stage of the persistent kernel 5.6); with many the operands that all SMs together draw from
// L2, 13 - 16 TB/s (gate/up of 768 rows: 282 MB in tiles of pairs, 453 MB in 128 x 128 ones), and under sustained load the power limit.  Measured
// with other operands on every launch, in turn with the stage of the persistent kernel: gate/up + GeGLU 768 x 32768 x 2048 33.5 us (43.6), BF16
// 333 x 1000 x 1152 6.4 (8.2), FP8 768 x 2048 x 16384 34.7 (42.7; without the split of K 34.2 - 43 by tile).
//
// CTAs stay for several tiles; where tensor memory holds two accumulators, the drain of one tile overlaps the MMAs of the next.
#pragma once
#include "op_gemm.cuh"
#include "solo.h"
#include "solo_common.cuh"

namespace pi0 {

struct SoloGemmCtl {
    uint64_t full[kSoloMaxSlots], empty[kSoloMaxSlots];
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem;
    int abort;
};

template <int OPERANDS, int EPI, int CG>
__global__ void __launch_bounds__(128 + 32 * solo_drain_warps(OPERANDS, EPI), 1) pi0_gemm_kernel(const __grid_constant__ SoloGemm p) {
    constexpr bool kScaled = OPERANDS == GEMM_NVFP4;
    constexpr int kDrainWarps = solo_drain_warps(OPERANDS, EPI), kShares = kDrainWarps / 4;     // draining warps, parts of a tile's columns
    constexpr int kC = CG == 2 ? kSoloChunks2 : kSoloChunks1;
    constexpr bool kLean = EPI == EPI_F32 && kScaled;        // (raw NVFP4 products: nothing is added)
    constexpr bool kResidual = EPI != EPI_GEGLU_FP4 && !kLean;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    SoloGemmCtl* ctl = reinterpret_cast<SoloGemmCtl*>(base);
    uint8_t* data = base + kSoloCtlBytes;
    const GemmParams& g = p.g;
    const int warp = threadIdx.x >> 5, lane = lane_id();
    const int quarter = warp & 3, share = (warp - 4) >> 2;    // (draining warps)
    const bool third = kScaled || p.b_boxes > 2;              // warp 2 copies too
    // A cluster is one pair per K split of a tile; in a pair the first CTA leads.
    const uint32_t cluster_place = CG == 2 ? cluster_rank() : 0u, first_rank = cluster_place & ~1u, rank = cluster_place - first_rank;
    const bool leader = rank == 0;
    const int split = static_cast<int>(cluster_place) / CG, group = CG * p.splits;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kSoloMaxSlots; s++) {
            mbar_init(&ctl->full[s], third ? 3 : 2);         // the leader's copying threads announce what they, and the other CTA's, bring
            mbar_init(&ctl->empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&ctl->acc_full[b], 1);
            mbar_init(&ctl->acc_empty[b], kDrainWarps * CG);
        }
        ctl->abort = 0;
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc_cg<CG>(&ctl->tmem, static_cast<uint32_t>(p.tmem_cols));
    if (warp == 0 && lane == 0) {
        prefetch_tmap(&p.map_a);
    }
    if (warp == 3 && lane == 0) prefetch_tmap(&p.map_b);
    if (kScaled && CG == 2 && warp == 2 && lane == 0) {
        prefetch_tmap(&p.map_sfa);
        prefetch_tmap(&p.map_sfb);
    }
    tc_fence_before();
    __syncthreads();
    if (CG == 2) cluster_sync();                             // the other CTA's barriers exist
    tc_fence_after();
    const uint32_t tmem = ctl->tmem;
    if (p.guard.early && warp == 4) {
        grid_dependency_wait();
        grid_launch_dependents();
    }
    const int unit = static_cast<int>(blockIdx.x) / group, units = static_cast<int>(gridDim.x) / group;
    const int items = p.items, m_tiles = p.m_tiles;
    const int ks_begin = p.slots * split / p.splits, ks_end = p.slots * (split + 1) / p.splits;
    const SoloWait w{p.guard.status, p.guard.budget_ns, &ctl->abort};

    // The copying threads and the issuing one keep all of their arguments in registers, fetched while the kernel in front still runs: each
    // has to pass on a slot in less time than its MMAs take (with divisions and constant loads in the loop a slot of a pair's tile took 570 -
    // 1,500 cycles, and gate/up in pairs of 192 columns 53 us; 31 from registers, 29 with three copying threads instead of two).
    if (warp == 0 || warp == 2 || warp == 3) {
        // (each copy costs the thread that sends it some 130 cycles: three of them share the up to six of a slot)
        if (lane == 0 && (warp != 2 || third)) {
            const uint32_t full0 = CG == 2 ? map_to_rank(smem_u32(&ctl->full[0]), first_rank) : smem_u32(&ctl->full[0]);
            const uint32_t stages = static_cast<uint32_t>(p.stages), stride = static_cast<uint32_t>(p.stride);
            const int k_groups = g.k_groups, tile_rows = p.tile_rows, bn = p.bn;
            uint32_t slot = 0, phase = 1;
            bool alive = true;
            if (warp == 0) {
                const uint32_t bytes = static_cast<uint32_t>(p.a_rows) * 128u * kC, off_sf = static_cast<uint32_t>(p.off_sfa);
                const void *map = &p.map_a, *map_sf = &p.map_sfa;
                const uint8_t* scales = g.sfa;
                grid_dependency_wait();
                for (int tile = unit; alive && tile < items; tile += units) {
                    const int m0 = (tile % m_tiles * CG + static_cast<int>(rank)) * tile_rows;
                    int atom = (m0 >> 7) * k_groups + ks_begin * 4 * kC, left = k_groups - ks_begin * 4 * kC;
#pragma unroll 1
                    for (int ks = ks_begin; ks < ks_end; ++ks) {
                        if (!solo_wait(w, &ctl->empty[slot], phase)) { alive = false; break; }
                        // (pairs bring whole groups of scale atoms by tensor map: beyond the last one the copy engine fills zeros)
                        const uint32_t sf = !kScaled ? 0u : 512u * (CG == 2 ? 4u * kC : static_cast<uint32_t>(min(4 * kC, left)));
                        if (leader) mbar_expect_tx(&ctl->full[slot], (bytes + sf) * CG);
                        uint8_t* dst = data + slot * stride;
                        tma_load_3d_cg<CG>(dst, map, full0 + slot * 8u, 0, m0, ks * kC);
                        if (kScaled) {
                            if (CG == 2) tma_load_2d_cg<CG>(dst + off_sf, map_sf, full0 + slot * 8u, 0, atom);
                            else bulk_load(dst + off_sf, scales + static_cast<size_t>(atom) * 512, sf, &ctl->full[slot]);
                            atom += 4 * kC;
                            left -= 4 * kC;
                        }
                        if (++slot == stages) { slot = 0; phase ^= 1u; }
                    }
                }
            } else {
                // B: at most four copies per chunk, two of them by each thread
                const uint32_t off_b = static_cast<uint32_t>(p.off_b), off_sfb = static_cast<uint32_t>(p.off_sfb);
                const int block = p.b_block, boxes = p.b_boxes, box_rows = p.b_rows, per_tile = p.sfb_per_tile, atoms = p.sfb_atoms;
                const int box0 = warp == 3 ? 0 : 2, mine = warp == 3 ? min(boxes, 2) : max(boxes - 2, 0);
                const uint32_t box_bytes = static_cast<uint32_t>(box_rows) * 128u * kC * static_cast<uint32_t>(mine);
                const void *map = &p.map_b, *map_sfb = &p.map_sfb;
                const uint8_t* sfb = g.sfb;
                grid_dependency_wait();
                for (int tile = unit; alive && tile < items; tile += units) {
                    const int n_tile = tile / m_tiles, n0 = n_tile * bn;
                    int at[2], blk[2];                                        // where a copy begins inside its block of rows, and which block that is
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        const int r = n0 + static_cast<int>(rank) * (bn / CG) + (box0 + b) * box_rows;
                        blk[b] = r / block;
                        at[b] = r - blk[b] * block;
                    }
                    const int b_atom = per_tile ? n_tile : n0 >> 7;
                    int atom = b_atom * k_groups + ks_begin * 4 * kC, left = k_groups - ks_begin * 4 * kC;
#pragma unroll 1
                    for (int ks = ks_begin; ks < ks_end; ++ks) {
                        if (!solo_wait(w, &ctl->empty[slot], phase)) { alive = false; break; }
                        uint8_t* dst = data + slot * stride;
                        const uint32_t bar = full0 + slot * 8u;
                        const uint32_t sf = !kScaled || warp == 3 ? 0u : 512u * (CG == 2 ? 4u * kC : static_cast<uint32_t>(min(4 * kC, left)));
                        if (leader) mbar_expect_tx(&ctl->full[slot], (box_bytes + sf * static_cast<uint32_t>(atoms)) * CG);
                        if (boxes == 1) {
                            if (mine) tma_load_4d_cg<CG>(dst + off_b, map, bar, 0, at[0], ks * kC, blk[0]);
                        } else {
#pragma unroll
                            for (int c = 0; c < kC; ++c)
#pragma unroll
                                for (int b = 0; b < 2; ++b)
                                    if (b < mine) tma_load_4d_cg<CG>(dst + off_b + (c * boxes + box0 + b) * box_rows * 128, map, bar, 0, at[b], ks * kC + c, blk[b]);
                        }
                        if (kScaled && warp == 2) {
                            if (CG == 2) tma_load_3d_cg<CG>(dst + off_sfb, map_sfb, bar, 0, ks * 4 * kC, b_atom);
                            else bulk_load(dst + off_sfb, sfb + static_cast<size_t>(atom) * 512, sf, &ctl->full[slot]);
                            atom += 4 * kC;
                            left -= 4 * kC;
                        }
                        if (++slot == stages) { slot = 0; phase ^= 1u; }
                    }
                }
            }
        }
    } else if (warp == 1) {
        // (values broadcast over the whole warp, in front of the election, stay in uniform registers, which the tcgen05 instructions want)
        constexpr uint64_t kOperandHi = (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
        constexpr uint64_t kScaleHi = (1ull << 16) | (8ull << 32) | (1ull << 46);
        const bool two_atoms = CG == 2 && uniform_i32(p.sfb_atoms) == 2;      // (tiles of more than 128 columns)
        const uint32_t tmem_u = uniform_u32(tmem), data16 = uniform_u32((smem_u32(data) & 0x3FFFFu) >> 4);
        const uint32_t a_chunk16 = uniform_u32(static_cast<uint32_t>(p.a_rows)) * 8u, b_chunk16 = uniform_u32(static_cast<uint32_t>(p.bn / CG)) * 8u;
        const uint32_t sfb_groups = two_atoms ? 8u : 4u, sf_slot = 4u * kC * (4u + sfb_groups);
        const uint32_t stages = uniform_u32(static_cast<uint32_t>(p.stages)), stride16 = uniform_u32(static_cast<uint32_t>(p.stride)) >> 4;
        const uint32_t off_b16 = uniform_u32(static_cast<uint32_t>(p.off_b)) >> 4, off_sfa16 = uniform_u32(static_cast<uint32_t>(p.off_sfa)) >> 4,
                       off_sfb16 = uniform_u32(static_cast<uint32_t>(p.off_sfb)) >> 4;
        const uint32_t sf_col = tmem_u + uniform_u32(static_cast<uint32_t>(p.sf_col)), sf_mask = uniform_u32(static_cast<uint32_t>(p.sf_mask)), idesc = uniform_u32(g.idesc);
        const uint32_t acc_stride = uniform_u32(static_cast<uint32_t>(p.acc_stride));
        const int k_groups = uniform_i32(g.k_groups), bn = uniform_i32(p.bn), ks_first = uniform_i32(ks_begin), ks_last = uniform_i32(ks_end);
        const bool per_tile = p.sfb_per_tile != 0, two_bufs = uniform_i32(p.acc_bufs) == 2;
        const uint16_t both = static_cast<uint16_t>(3u << uniform_u32(first_rank));
        if (leader && elect_one()) {
            uint32_t slot = 0, phase = 0, use = 0, it = 0;
            bool alive = true, landed = false;                                // landed: the slot was seen full half-way through the one before
            for (int tile = unit; alive && tile < items; tile += units) {
                const uint32_t buf = two_bufs ? use & 1u : 0u, acc_phase = (two_bufs ? use >> 1 : use) & 1u;
                if (!solo_wait_cluster<CG>(w, &ctl->acc_empty[buf], acc_phase ^ 1u)) break;
                tc_fence_after();
                const uint32_t d = tmem_u + buf * acc_stride;
                const uint32_t sub = per_tile ? 0u : static_cast<uint32_t>((tile / m_tiles * bn) & 127) >> 5;    // (even: tiles are multiples of 64 columns)
#pragma unroll 1
                for (int ks = ks_first; ks < ks_last; ++ks) {
                    if (!landed && !solo_wait(w, &ctl->full[slot], phase)) { alive = false; break; }
                    const uint32_t next = slot + 1 == stages ? 0u : slot + 1, next_phase = next == 0 ? phase ^ 1u : phase;
                    const uint32_t a16 = data16 + slot * stride16, b16 = a16 + off_b16;
                    const uint32_t groups = static_cast<uint32_t>(min(4 * kC, k_groups - ks * 4 * kC));
                    const uint32_t sfa = sf_col + (it & sf_mask) * sf_slot, sfb = sfa + 16u * kC;
                    const uint32_t sfa16 = a16 + off_sfa16, sfb16 = a16 + off_sfb16;
                    auto copy_scales = [&](uint32_t gi, bool two) {
                        tc_copy_sf_cg<CG>(sfa + gi * 4, kScaleHi | static_cast<uint64_t>(sfa16 + gi * 32));
                        tc_copy_sf_cg<CG>(sfb + gi * (two ? 8u : 4u), kScaleHi | static_cast<uint64_t>(sfb16 + gi * 32));
                        if (two) tc_copy_sf_cg<CG>(sfb + gi * 8 + 4, kScaleHi | static_cast<uint64_t>(sfb16 + 4 * kC * 32 + gi * 32));
                    };
                    auto issue = [&](uint32_t gi, uint32_t acc) {
                        const uint32_t chunk = gi >> 2, k32 = gi & 3u;
                        const uint64_t da = kOperandHi | static_cast<uint64_t>(a16 + chunk * a_chunk16 + 2u * k32);
                        const uint64_t db = kOperandHi | static_cast<uint64_t>(b16 + chunk * b_chunk16 + 2u * k32);
                        if constexpr (OPERANDS == GEMM_NVFP4) tc_mma_nvfp4_cg<CG>(d, da, db, idesc, sfa + gi * 4, sfb + gi * sfb_groups + sub, acc);
                        else tc_mma_dense_cg<CG, OPERANDS == GEMM_FP8>(d, da, db, idesc, acc);
                    };
                    if (groups == 4u * kC) {
                        // (all scale copies in front of the MMAs: alternating costs the tensor pipe)
                        if constexpr (kScaled) {
                            if (two_atoms) {
#pragma unroll
                                for (uint32_t gi = 0; gi < 4u * kC; ++gi) copy_scales(gi, true);
                            } else {
#pragma unroll
                                for (uint32_t gi = 0; gi < 4u * kC; ++gi) copy_scales(gi, false);
                            }
                        }
#pragma unroll
                        for (uint32_t gi = 0; gi < 4u * kC; ++gi) {
                            if (gi == 2u * kC) landed = mbar_test_wait(&ctl->full[next], next_phase);
                            issue(gi, gi != 0 ? 1u : static_cast<uint32_t>(ks != ks_first));
                        }
                    } else {
                        landed = false;
#pragma unroll 1
                        for (uint32_t gi = 0; gi < groups; ++gi) {
                            if constexpr (kScaled) copy_scales(gi, two_atoms);
                            issue(gi, static_cast<uint32_t>(ks != ks_first || gi != 0));
                        }
                    }
                    tc_commit_cg<CG>(&ctl->empty[slot], both);
                    slot = next;
                    phase = next_phase;
                    ++it;
                }
                if (alive) tc_commit_cg<CG>(&ctl->acc_full[buf], both);
                ++use;
            }
        }
    } else if (warp >= 4) {
        uint32_t use = 0;
        grid_dependency_wait();
        for (int tile = unit; tile < items; tile += units, ++use) {
            const uint32_t buf = p.acc_bufs == 2 ? use & 1u : 0u, acc_phase = (p.acc_bufs == 2 ? use >> 1 : use) & 1u;
            const int n_tile = tile / m_tiles;
            const int m0 = ((tile - n_tile * m_tiles) * CG + static_cast<int>(rank)) * p.tile_rows, n0 = n_tile * p.bn;
            const int row = m0 + quarter * 32 + lane;
            const bool rows_here = quarter * 32 < p.tile_rows && m0 + quarter * 32 < g.rows, row_ok = row < g.rows;
            const int parts = min(p.bn, g.cols - n0) >> 5;                    // (logical columns are multiples of 32)
            const int col_begin = parts * share / kShares * 32, col_end = parts * (share + 1) / kShares * 32;
            const bool work = rows_here && col_begin < col_end;
            const DrainRow d = drain_row<EPI, kLean>(g, row);
            uint4 res[4] = {};
            auto load_residual = [&](int c) {
                if (kResidual && d.residual && row_ok) {
                    const uint4* r = reinterpret_cast<const uint4*>(d.residual + (n0 + c) * 2);
#pragma unroll
                    for (int i = 0; i < 4; i++) res[i] = __ldcg(r + i);
                }
            };
            if (work) load_residual(col_begin);                               // (on its way while the MMAs run)
            if (work && kResidual && d.bias && lane * 64 < (col_end - col_begin)) prefetch_l1(d.bias + (n0 + col_begin) * 2 + lane * 128);
            if (!solo_wait_warp(w, &ctl->acc_full[buf], acc_phase)) break;
            if (p.splits > 1) break;                                          // (one tile; drained below, by the pairs together)
            tc_fence_after();
            const uint32_t taddr = tmem + buf * static_cast<uint32_t>(p.acc_stride) + (static_cast<uint32_t>(quarter * 32) << 16);
            auto columns_read = [&]() {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (leader) mbar_arrive(&ctl->acc_empty[buf]);
                    else mbar_arrive_remote(map_to_rank(smem_u32(&ctl->acc_empty[buf]), first_rank));
                }
            };
            if (!work) {
                columns_read();
                continue;
            }
            float2 unused_a = make_float2(0.f, 0.f), unused_b = make_float2(0.f, 0.f);
#pragma unroll 1
            for (int c = col_begin; c < col_end; c += 32) {
                uint32_t raw[32];
                tmem_ld32(taddr + c, raw);
                tmem_ld_wait();
                if (c + 32 >= col_end) columns_read();
                gemm_epilogue_chunk<EPI, kLean, true>(g, d, raw, res, row, n0 + c, row_ok, g.alpha, 0.f, unused_a, unused_b);
                if (c + 32 < col_end) load_residual(c + 32);
            }
            if (warp == kDrainWarps && lane == 0) atomicAdd(p.guard.counters + (m0 >> 7), solo_gave_up(&ctl->abort) ? 0u : 1u);     // (quarter 0, the last columns)
        }
    }

    if constexpr (CG == 2 && !kScaled) {
        // K split over the pairs of a cluster: each pair has summed a part of K for the whole tile.  Pair s takes a share of the 32-column
        // pieces; the others leave theirs in its shared memory, which nobody copies into any more, and it adds them in the order of the
        // splits, its own from tensor memory.
        if (p.splits > 1) {
            const int n_tile = unit / m_tiles;
            const int m0 = ((unit - n_tile * m_tiles) * CG + static_cast<int>(rank)) * p.tile_rows, n0 = n_tile * p.bn;
            const int parts = min(p.bn, g.cols - n0) >> 5;
            const uint32_t taddr = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && solo_gave_up(&ctl->abort))                       // a part of the sum is missing: the tile is nobody's
                for (int r = 0; r < group; ++r) st_cluster_int(map_to_rank(smem_u32(&ctl->abort), static_cast<uint32_t>(r)), 1);
            cluster_sync();                                                   // all MMAs of the cluster are done
            const bool whole = !solo_gave_up(&ctl->abort), work = whole && warp >= 4 && m0 + quarter * 32 < g.rows;
            tc_fence_after();
            if (work) {
#pragma unroll 1
                for (int s = 0; s < p.splits; ++s) {
                    if (s == split) continue;
                    const int first = parts * s / p.splits, end = parts * (s + 1) / p.splits;
                    const int from = split < s ? split : split - 1;           // (place among the others)
#pragma unroll 1
                    for (int c = first + share; c < end; c += kShares) {
                        uint32_t raw[32];
                        tmem_ld32(taddr + c * 32, raw);
                        tmem_ld_wait();
                        const uint32_t dst = map_to_rank(smem_u32(data) + ((((c - first) * (p.splits - 1) + from) * 4 + quarter) * 256 + lane) * 16,
                                                         static_cast<uint32_t>(s * CG) + (cluster_place & 1u));
#pragma unroll
                        for (int i = 0; i < 8; i++) st_cluster_v4(dst + i * 512, raw[4 * i], raw[4 * i + 1], raw[4 * i + 2], raw[4 * i + 3]);
                    }
                }
            }
            __syncwarp();
            cluster_sync();                                                   // all partial sums have arrived
            if (work) {
                const int row = m0 + quarter * 32 + lane;
                const bool row_ok = row < g.rows;
                const DrainRow d = drain_row<EPI, kLean>(g, row);
                const int first = parts * split / p.splits, end = parts * (split + 1) / p.splits;
                float2 unused_a = make_float2(0.f, 0.f), unused_b = make_float2(0.f, 0.f);
#pragma unroll 1
                for (int c = first + share; c < end; c += kShares) {
                    uint4 res[4] = {};
                    if (d.residual && row_ok) {
                        const uint4* r = reinterpret_cast<const uint4*>(d.residual + (n0 + c * 32) * 2);
#pragma unroll
                        for (int i = 0; i < 4; i++) res[i] = __ldcg(r + i);
                    }
                    uint32_t raw[32];
                    float sum[32];
                    tmem_ld32(taddr + c * 32, raw);
                    tmem_ld_wait();
#pragma unroll 1
                    for (int s = 0; s < p.splits; ++s) {
                        const int from = s < split ? s : s - 1;
                        const float4* src = reinterpret_cast<const float4*>(data) + (((c - first) * (p.splits - 1) + from) * 4 + quarter) * 256 + lane;
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            const float4 q = s == split ? make_float4(__uint_as_float(raw[4 * i]), __uint_as_float(raw[4 * i + 1]), __uint_as_float(raw[4 * i + 2]),
                                                                      __uint_as_float(raw[4 * i + 3])) : src[i * 32];
                            sum[4 * i] = s == 0 ? q.x : sum[4 * i] + q.x;
                            sum[4 * i + 1] = s == 0 ? q.y : sum[4 * i + 1] + q.y;
                            sum[4 * i + 2] = s == 0 ? q.z : sum[4 * i + 2] + q.z;
                            sum[4 * i + 3] = s == 0 ? q.w : sum[4 * i + 3] + q.w;
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 32; i++) raw[i] = __float_as_uint(sum[i]);
                    gemm_epilogue_chunk<EPI, kLean, true>(g, d, raw, res, row, n0 + c * 32, row_ok, g.alpha, 0.f, unused_a, unused_b);
                }
            }
            if (whole && warp == 4 && lane == 0 && split == 0 && m0 < g.rows) atomicAdd(p.guard.counters + (m0 >> 7), 1u);
        }
    }

    // Everybody meets here: every wait above is bounded.  After one that ran out, copies in flight get a moment to land.
    __syncwarp();
    if (solo_gave_up(&ctl->abort)) {
        const unsigned long long t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (CG == 2) cluster_sync();
    tc_fence_after();
    if (warp == 1) tmem_dealloc_cg<CG>(tmem, static_cast<uint32_t>(p.tmem_cols));
}

template <int OPERANDS, int EPI, int CG>
cudaError_t launch_solo_gemm_form(const SoloGemm& p, int grid, size_t smem, cudaStream_t stream) {
    static bool configured[64] = {};
    const auto kernel = pi0_gemm_kernel<OPERANDS, EPI, CG>;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    if (device >= 64 || !configured[device]) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSoloDataBytes + kSoloCtlBytes + 1024);
        if (e != cudaSuccess) return e;
        if (device < 64) configured[device] = true;
    }
    cudaLaunchAttribute attrs[2] = {};
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = CG * p.splits;
    attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(grid);
    config.blockDim = dim3(128 + 32 * solo_drain_warps(OPERANDS, EPI));
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = attrs;
    config.numAttrs = CG == 2 ? 2 : 1;
    return cudaLaunchKernelEx(&config, kernel, p);
}

}  // namespace pi0
