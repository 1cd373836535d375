// GEMM instruction:  out[M,N] = epilogue(alpha * A[M,K] . B[N,K]^T), FP32 accumulation in tensor memory.
// Operands: NVFP4 (packed E2M1 with E4M3 block scales, tcgen05.mma kind::mxf4nvf4.block_scale), BF16 (kind::f16) or
// FP8 E4M3 (kind::f8f6f4).  In every format a row of K is cut into 128-byte chunks and one MMA consumes 32 bytes of
// each operand row (64 FP4, 16 BF16 or 32 FP8 elements), so the copy ring and the issue loop are the same code.
//
//   warps 0 and 3   : TMA producers - A and B tiles (128 B swizzled rows) and their scale atoms into a ring of slots; the
//                                     ring is laid out per GEMM: 3 slots of 72 KiB for 128-wide NVFP4 tiles, up to 5 for narrow
//                                     ones, up to 8 for dense operands (so slots of one size can come in different numbers)
//   warp 1          : MMA issuer    - one elected thread issues tcgen05.cp (scales smem->TMEM, NVFP4 only) and
//                                     tcgen05.mma, 32 operand bytes of K each
//   warps 4..7      : epilogue      - tcgen05.ld of a 128xN FP32 accumulator (one row per thread), fused math, stores
//   warps 0..3      : second half of the columns of an instruction's last tile, once their roles are done
//
// Two TMEM accumulators alternate, so the epilogue of tile t overlaps the MMAs of tile t+1 (192-wide tiles take both). Pipeline positions live in
// registers (PipeState) and carry over from one instruction to the next; barriers are never re-initialised.
#pragma once
#include "vm_core.cuh"

namespace pi0 {

// The copy warps: warp 0 (WEIGHTS = false) brings A and its scales, warp 3 (WEIGHTS = true) B and its scales; lane 0 of
// each issues the copies and every slot's barrier expects one arrival from both.
//
// Weights never depend on another stage, so warp 3 takes no part in the dependency wait: it fills whatever slots are free,
// also those of the next GEMM instruction, and when the producers are done only the activation half is still to be
// fetched.  One warp issuing all four copies of a slot (each costs the issuing thread about 65 cycles) was as slow as the
// MMAs that read it.
// The loop works on register copies of the descriptor: that lies in shared memory, and every asm statement with a memory
// clobber would make the compiler read it again.
// WIDE: also the two scale atoms per group of 192-wide tiles.  With that choice in its loop the copy warp of a few-row projection is later
// (q|k|v of 51 rows 5.65 -> 5.76 us), so the lean variant without such tiles goes without; the ones with every operator keep
// it, where nothing was gained (BF16 forward 16.13 ms without, 16.08 with).
template <bool WEIGHTS, bool WIDE>
__device__ __forceinline__ void gemm_producer(const VmProgram& prog, Ctl* ctl, uint8_t* data, const StageDesc& st,
                                              int stage_index, int first, int count, PipeState& ps, long long* stamp) {
    const GemmParams& g = st.p.gemm;
    const int lane = lane_id();
    uint32_t slot = ps.slot, bits = ps.bits;
    const int k_groups = g.k_groups, n_tiles = g.n_tiles, block_n = g.block_n, b_tiled = g.b_tiled;
    const void* tmap = WEIGHTS ? g.tmap_b : g.tmap_a;
    const uint8_t* scales = WEIGHTS ? g.sfb : g.sfa;
    const int chunks = (k_groups + 3) >> 2;                          // 256-wide K chunks
    const int slots = (chunks + kChunks - 1) / kChunks;
    const uint32_t bytes = static_cast<uint32_t>(kChunks) * 128u * static_cast<uint32_t>(WEIGHTS ? block_n : g.a_box_rows);
    const uint32_t ring = static_cast<uint32_t>(g.ring_stages), stride = static_cast<uint32_t>(g.slot_stride);
    const uint32_t off = WEIGHTS ? static_cast<uint32_t>(g.off_b) : 0u, off_sf = static_cast<uint32_t>(WEIGHTS ? g.off_sfb : g.off_sfa);
    const bool scaled = g.operands == GEMM_NVFP4;                    // scale atoms: 512 bytes per MMA group and operand
    const uint32_t geo = ring_key(g.slot_stride, g.ring_stages);
    if (ps.geo != geo) {
        // Slots of the previous geometry overlap the new ones at other indices, or are more than the new ring has: every copy issued so far must have
        // been read by its MMAs before the first new copy lands (waits for the last release of each slot).
        int alive0 = 1;
        if (lane == 0 && ps.geo != 0)                           // (nothing to wait for in front of the first GEMM)
            for (int s = 0; s < kMaxStagesDense && alive0; ++s)
                alive0 = mbar_wait(prog, ctl, &ctl->empty[s], ((bits >> s) & 1u) ^ 1u, stage_index) ? 1 : 0;
        alive0 = __shfl_sync(0xffffffffu, alive0, 0);
        if (!alive0) return;
        ps.geo = geo;
        slot = 0;
    }
    int current_band = -1;
    for (int t = first; t < first + count; ++t) {
        const int m_tile = t / n_tiles, n_tile = t - m_tile * n_tiles;
        if (!WEIGHTS) {
            const int band = tile_band(st, t);
            if (band != current_band) {
                if (!warp_wait_sources(prog, ctl, st, stage_index, band, band)) return;
                if (lane == 0) {
                    fence_proxy_async_global();
                    if (current_band < 0) word_set(&ctl->deps_seen, ps.gemm_seq + 1u);   // tell the draining warps: the sources of this instruction's first band are complete
                    if (stamp && current_band < 0) stamp[1] = static_cast<long long>(global_ns());
                }
                current_band = band;
            }
        }
        int alive = 1;
        if (lane == 0) {
            // B scales: the 128-row atom that holds the tile's rows, or - 32- and 192-wide tiles - an atom or two of the tile's own
            const bool two = WIDE && WEIGHTS && block_n > 128;
            const int sf_tile = !WEIGHTS ? m_tile : block_n == 32 ? n_tile : two ? 2 * n_tile : (n_tile * block_n) >> 7;
            const uint32_t sf_group = two ? 1024u : 512u;
            const uint8_t* sf = scales + static_cast<size_t>(sf_tile) * k_groups * 512;
            for (int ks = 0; ks < slots; ++ks) {
                const uint32_t s = slot;
                if (!mbar_wait(prog, ctl, &ctl->empty[s], ((bits >> s) & 1u) ^ 1u, stage_index)) { alive = 0; break; }
                uint8_t* base = data + s * stride;
                uint64_t* bar = &ctl->full[s];
                const uint32_t sf_bytes = scaled ? static_cast<uint32_t>(min(4 * kChunks, k_groups - ks * 4 * kChunks)) * sf_group : 0u;
                // Boxes always deliver kChunks chunks (beyond K the copy engine fills zeros or, inside a padded
                // allocation, bytes that no MMA reads).  a_box_rows < 128 (few logical rows): only the rows that
                // exist are copied; the MMA still reads 128 rows, the rest lands in accumulator rows never stored.
                mbar_expect_tx(bar, bytes + sf_bytes);
                if (WEIGHTS && b_tiled) tma_load_2d(base + off, tmap, bar, 0, (n_tile * chunks + ks * kChunks) * block_n);
                else tma_load_3d(base + off, tmap, bar, 0, WEIGHTS ? n_tile * block_n : m_tile * 128, ks * kChunks);
                if (scaled) bulk_load(base + off_sf, sf + static_cast<size_t>(ks) * (4 * kChunks) * sf_group, sf_bytes, bar);
                bits ^= 1u << s;
                slot = s + 1 == ring ? 0u : s + 1;
            }
        }
        alive = __shfl_sync(0xffffffffu, alive, 0);
        if (!alive) return;
    }
    ps.slot = slot;
    ps.bits = bits;
}

// The issuing thread's loop for NVFP4 tiles of 192 columns.  Such a tile takes both accumulator buffers (two uses) from column 0 on and
// has two atoms of B scales per group, so the scale columns of a slot are A's four of every group (eight apart) and behind them B's
// eight, two slots in turn.  It is the one tile of its instruction as a rule; the loop of the other widths stays free of it (with
// the place of the scale columns as a variable, or both widths from one template, a slot takes 40 - 100 ns longer).
__device__ __forceinline__ void gemm_mma_wide(const VmProgram& prog, Ctl* ctl, const GemmParams& g, uint32_t data16, uint32_t tmem, int stage_index,
                                              int count, uint32_t& slot, uint32_t& bits, uint32_t& it, uint32_t& tile_no, long long* stamp) {
    constexpr uint64_t kOperandHi = (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
    constexpr uint64_t kScaleHi = (1ull << 16) | (8ull << 32) | (1ull << 46);
    const int k_groups = g.k_groups, slots = (k_groups + 4 * kChunks - 1) / (4 * kChunks);
    const uint32_t a_chunk16 = static_cast<uint32_t>(g.a_box_rows) * 8u, b_chunk16 = static_cast<uint32_t>(g.block_n) * 8u;
    for (int t = 0; t < count; ++t) {
        for (uint32_t u = 0; u < 2; ++u)
            if (!mbar_wait(prog, ctl, &ctl->acc_empty[(tile_no + u) & 1u], (((tile_no + u) >> 1) & 1u) ^ 1u, stage_index)) return;
        tc_fence_after();
        for (int ks = 0; ks < slots; ++ks) {
            if (!mbar_wait(prog, ctl, &ctl->full[slot], (bits >> slot) & 1u, stage_index)) return;
            if (stamp && t == 0 && ks == 0) stamp[4] = static_cast<long long>(global_ns());
            const uint32_t a16 = data16 + (slot * static_cast<uint32_t>(g.slot_stride) >> 4), b16 = a16 + (static_cast<uint32_t>(g.off_b) >> 4);
            const uint32_t sfa16 = a16 + (static_cast<uint32_t>(g.off_sfa) >> 4), sfb16 = a16 + (static_cast<uint32_t>(g.off_sfb) >> 4);
            const uint32_t groups = static_cast<uint32_t>(min(4 * kChunks, k_groups - ks * 4 * kChunks));
            const uint32_t sfa = tmem + kSfCol0 + (it & 1u) * 128u, sfb = sfa + 64u;
            for (uint32_t gi = 0; gi < groups; ++gi) {
                tc_copy_sf(sfa + gi * 8, kScaleHi | static_cast<uint64_t>(sfa16 + gi * 32));
                tc_copy_sf(sfb + gi * 8, kScaleHi | static_cast<uint64_t>(sfb16 + gi * 64));
                tc_copy_sf(sfb + gi * 8 + 4, kScaleHi | static_cast<uint64_t>(sfb16 + gi * 64 + 32));
            }
            for (uint32_t gi = 0; gi < groups; ++gi) {
                const uint32_t chunk = gi >> 2, sub = gi & 3u;
                tc_mma_nvfp4(tmem, kOperandHi | static_cast<uint64_t>(a16 + chunk * a_chunk16 + 2u * sub),
                             kOperandHi | static_cast<uint64_t>(b16 + chunk * b_chunk16 + 2u * sub), g.idesc, sfa + gi * 8, sfb + gi * 8,
                             static_cast<uint32_t>(ks != 0 || gi != 0));
            }
            tc_commit(&ctl->empty[slot]);
            bits ^= 1u << slot;
            slot = slot + 1 == static_cast<uint32_t>(g.ring_stages) ? 0u : slot + 1;
            it++;
        }
        tc_commit(&ctl->acc_full[0]);
        tc_commit(&ctl->acc_full[1]);
        tile_no += 2;
    }
}

// Warp 1: one elected thread runs the whole loop - waits, scale copies, MMAs, commits - while the other lanes wait at the
// end.  The queue in front of the tensor core holds only about two MMAs, so whatever the issuing thread does between two
// slots is idle tensor time: with a warp-wide barrier vote and an election per slot a slot of eight MMAs cost 690 (BF16,
// 32 columns) to 1050 cycles (NVFP4, 128 columns), alone it needs 325 and 740.  The barrier of the next slot is therefore
// tested (without blocking) half-way through the current one, and a slot that has landed by then costs no wait at all.
// The operand arithmetic starts from values broadcast over the warp, so that descriptors stay in uniform registers.
// (One instantiation per operand format, so each issue loop carries only its own instructions.)
template <int OPERANDS, bool WIDE>
__device__ __forceinline__ void gemm_mma(const VmProgram& prog, Ctl* ctl, uint8_t* data, uint32_t tmem_in, const StageDesc& st,
                                         int stage_index, int first_in, int count_in, PipeState& ps, long long* stamp) {
    const GemmParams& g = st.p.gemm;
    const int first = uniform_i32(first_in), count = uniform_i32(count_in);
    const int k_groups = uniform_i32(g.k_groups), n_tiles = uniform_i32(g.n_tiles), block_n = uniform_i32(g.block_n);
    const int chunks = (k_groups + 3) >> 2;
    const int slots = (chunks + kChunks - 1) / kChunks;
    const uint32_t a_chunk16 = uniform_u32(static_cast<uint32_t>(g.a_box_rows)) * 8u, b_chunk16 = static_cast<uint32_t>(block_n) * 8u;   // 16-byte units
    const uint32_t ring = uniform_u32(static_cast<uint32_t>(g.ring_stages)), stride = uniform_u32(static_cast<uint32_t>(g.slot_stride));
    const uint32_t off_b16 = uniform_u32(static_cast<uint32_t>(g.off_b)) >> 4, off_sfa16 = uniform_u32(static_cast<uint32_t>(g.off_sfa)) >> 4,
                   off_sfb16 = uniform_u32(static_cast<uint32_t>(g.off_sfb)) >> 4;
    const uint32_t idesc = uniform_u32(g.idesc);
    const uint32_t tmem = uniform_u32(tmem_in);
    const uint32_t data16 = uniform_u32((smem_u32(data) & 0x3FFFFu) >> 4), stride16 = stride >> 4;
    // descriptor high words: K-major 128-byte swizzle (8-row groups 1024 bytes apart, version 1) and the scale atoms
    // (no swizzle, 8-line groups 128 bytes apart)
    constexpr uint64_t kOperandHi = (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
    constexpr uint64_t kScaleHi = (1ull << 16) | (8ull << 32) | (1ull << 46);
    const uint32_t geo = ring_key(g.slot_stride, g.ring_stages);
    if (ps.geo != geo) { ps.geo = geo; ps.slot = 0; }
    uint32_t slot = uniform_u32(ps.slot), bits = uniform_u32(ps.bits), it = uniform_u32(ps.it), tile_no = uniform_u32(ps.tile);
    const bool leader = elect_one();
    if (WIDE && __builtin_expect(block_n > 128, 0)) {
        if (leader) gemm_mma_wide(prog, ctl, g, data16, tmem, stage_index, count, slot, bits, it, tile_no, stamp);
    } else if (leader) {
        bool landed = false, alive = true;                   // landed: the current slot was seen full by the look-ahead
        for (int t = first; alive && t < first + count; ++t) {
            const int n_tile = t % n_tiles;
            const uint32_t buf = tile_no & 1u, acc_phase = (tile_no >> 1) & 1u;
            if (!mbar_wait(prog, ctl, &ctl->acc_empty[buf], acc_phase ^ 1u, stage_index)) break;
            tc_fence_after();
            const uint32_t d = tmem + buf * 128u;
            // Scale rows of a 64-wide B tile sit in the 32-row sub-columns 0 or 2 of their 128-row atom (the scale operand of
            // the MMA must start at an even sub-column); 32-wide tiles bring atoms of their own with the rows in sub-column 0.
            const uint32_t sfb_sub = block_n == 32 ? 0u : static_cast<uint32_t>((n_tile * block_n) & 127) >> 5;
            for (int ks = 0; ks < slots; ++ks) {
                const uint32_t s = slot, next = s + 1 == ring ? 0u : s + 1;
                if (!landed && !mbar_wait(prog, ctl, &ctl->full[s], (bits >> s) & 1u, stage_index)) { alive = false; break; }
                if (stamp && t == first && ks == 0) stamp[4] = static_cast<long long>(global_ns());
                const int groups = min(4 * kChunks, k_groups - ks * 4 * kChunks);
                const uint32_t a16 = data16 + s * stride16;
                const uint32_t sf_cols = tmem + kSfCol0 + (it & 3u) * (4 * kChunks * 8);
                // Scales of group gi: smem -> tensor memory.  All copies of a slot are issued in front of its MMAs: alternating
                // between the two kinds of instruction costs the tensor pipe about 20 cycles per group (slots of 8 groups,
                // 128 x 32 / 64 / 128 tiles: 650 / 700 / 790 cycles alternating, 470 / 515 / 640 copies first).
                auto copy_scales = [&](uint32_t gi) {
                    tc_copy_sf(sf_cols + gi * 8, kScaleHi | static_cast<uint64_t>(a16 + off_sfa16 + gi * 32));
                    tc_copy_sf(sf_cols + gi * 8 + 4, kScaleHi | static_cast<uint64_t>(a16 + off_sfb16 + gi * 32));
                };
                auto issue = [&](uint32_t gi, uint32_t acc) {
                    const uint32_t chunk = gi >> 2, sub = gi & 3u;
                    // 64 FP4, 16 BF16 or 32 FP8 elements = 32 bytes along K inside the 128-byte swizzled row: advance the start
                    // address by 2 units
                    const uint64_t da = kOperandHi | static_cast<uint64_t>(a16 + chunk * a_chunk16 + 2u * sub);
                    const uint64_t db = kOperandHi | static_cast<uint64_t>(a16 + off_b16 + chunk * b_chunk16 + 2u * sub);
                    if constexpr (OPERANDS == GEMM_NVFP4) tc_mma_nvfp4(d, da, db, idesc, sf_cols + gi * 8, sf_cols + gi * 8 + 4 + sfb_sub, acc);
                    else if constexpr (OPERANDS == GEMM_BF16) tc_mma_f16(d, da, db, idesc, acc);
                    else tc_mma_f8(d, da, db, idesc, acc);
                };
                if (groups == 4 * kChunks) {                 // a full slot: no branch between its MMAs
                    if constexpr (OPERANDS == GEMM_NVFP4) {
#pragma unroll
                        for (uint32_t gi = 0; gi < 4 * kChunks; ++gi) copy_scales(gi);
                    }
#pragma unroll
                    for (uint32_t gi = 0; gi < 4 * kChunks; ++gi) {
                        if (gi == 2 * kChunks) landed = mbar_test_wait(&ctl->full[next], (bits >> next) & 1u);
                        issue(gi, gi != 0 ? 1u : static_cast<uint32_t>(ks != 0));
                    }
                } else {
                    landed = false;
#pragma unroll 1
                    for (uint32_t gi = 0; gi < static_cast<uint32_t>(groups); ++gi) {
                        if constexpr (OPERANDS == GEMM_NVFP4) copy_scales(gi);
                        issue(gi, static_cast<uint32_t>(ks != 0 || gi != 0));
                    }
                }
                tc_commit(&ctl->empty[s]);     // slot reusable once these MMAs have read it
                bits ^= 1u << s;
                slot = next;
                it++;
            }
            if (alive) tc_commit(&ctl->acc_full[buf]);    // accumulator complete
            tile_no++;
        }
    }
    __syncwarp();
    const int from = __ffs(__ballot_sync(0xffffffffu, leader)) - 1;
    ps.slot = __shfl_sync(0xffffffffu, slot, from);
    ps.bits = __shfl_sync(0xffffffffu, bits, from);
    ps.it = __shfl_sync(0xffffffffu, it, from);
    if (stamp && lane_id() == 0) stamp[5] = static_cast<long long>(global_ns());
}

// ---- epilogue helpers ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpack_bf16x2(uint32_t u) {
    __nv_bfloat162 h = *reinterpret_cast<__nv_bfloat162*>(&u);
    return __bfloat1622float2(h);
}
__device__ __forceinline__ float gelu_sigmoid(float x) {
    // x * sigmoid(2u), u = sqrt(2/pi)(x + 0.044715 x^3): identical to the tanh form.
    float z = 1.5957691216057308f * x * (1.f + 0.044715f * x * x);
    return __fdividef(x, 1.f + __expf(-z));
}

__device__ __forceinline__ void add_bf16x32(float2 (&v)[16], const uint4 (&u)[4]) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
        v[4 * i + 0] = add2(v[4 * i + 0], unpack_bf16x2(u[i].x));
        v[4 * i + 1] = add2(v[4 * i + 1], unpack_bf16x2(u[i].y));
        v[4 * i + 2] = add2(v[4 * i + 2], unpack_bf16x2(u[i].z));
        v[4 * i + 3] = add2(v[4 * i + 3], unpack_bf16x2(u[i].w));
    }
}
// NVFP4 codes of 32 values times inv_gs (16 bytes) and the two block scales in one word.
__device__ __forceinline__ uint4 quantize_32(const float2 (&v)[16], float inv_gs, uint32_t& codes) {
    uint32_t words[4];
    codes = 0;
#pragma unroll
    for (int half = 0; half < 2; half++) {
        float2 h[8];
#pragma unroll
        for (int i = 0; i < 8; i++) h[i] = mul2(v[8 * half + i], make_float2(inv_gs, inv_gs));
        uint32_t code;
        const uint2 bytes = quantize_block16(h, 0, code);
        words[2 * half] = bytes.x;
        words[2 * half + 1] = bytes.y;
        codes |= code << (8 * half);
    }
    return make_uint4(words[0], words[1], words[2], words[3]);
}
// What the drain of one accumulator row needs of the descriptor, in registers and with the row's offsets applied.  The
// descriptor lies in shared memory, and every asm statement with a memory clobber makes the compiler read a field again: a dozen
// dependent reads per chunk, from a shared memory that the MMAs keep busy (pi0 forward 9.22 -> 9.06 ms).
// (Only the fields that an epilogue kind uses exist in its drain.)
struct DrainRow {
    uint8_t* out;                // the row of the output
    const uint8_t* residual;     // the row of the residual, or null
    const uint8_t* bias;         // BF16 [N] or null
    const float* center;         // FP32 [N] or null
    uint8_t* copy;               // EPI_STREAM: the row of the NVFP4 copy
    uint8_t* scales;             // the row's place in the first scale atom of its row band
    float inv_gs;
    int ldo;                     // BF16 rows: bytes from one row of the output to the next
    int rows_left;               // rows from the warp's first one on
    int act, sums;
    bool together;               // EPI_QKV_ROPE: the warp stores its rows together (store_rows64)
};
// Scale of block `block` of that row (scale_offset, split into a part per row and a part per block).
__device__ __forceinline__ uint8_t* scale_at(const DrainRow& d, int block) { return d.scales + (block >> 2) * 512 + (block & 3); }
template <int EPI, bool LEAN>
__device__ __forceinline__ DrainRow drain_row(const GemmParams& g, int row) {
    DrainRow d = {};
    const int lane = lane_id();
    const size_t width = EPI == EPI_F32 ? 4 : EPI == EPI_FP4 || EPI == EPI_GEGLU_FP4 ? 1 : 2;
    d.ldo = g.ldo * 2;
    d.out = static_cast<uint8_t*>(g.out) + static_cast<size_t>(row) * g.ldo * width;
    d.rows_left = g.rows - (row - lane);
    constexpr bool kPlain = EPI == EPI_F32 && LEAN;              // (nothing is added)
    if (!kPlain && g.residual) d.residual = static_cast<const uint8_t*>(g.residual) + static_cast<size_t>(row) * g.ldr * 2;
    if (!kPlain) d.bias = static_cast<const uint8_t*>(g.bias);
    d.center = g.col_center;
    d.inv_gs = g.out_inv_gs;
    d.act = g.act;
    d.sums = g.sum_out != nullptr;
    // Row by row a store touches 32 lines, and the load / store unit takes one line a cycle: with eight warps at work (several row
    // bands) a Q | K | V drain waits for it; few rows keep two to four warps busy, and there the transposition only lengthens the
    // chain of a thread.  With the pair-major table below, q|k|v of the 768-row prefix 12.1 -> 9.4 us.
    d.together = g.rows > 128;
    if (EPI == EPI_STREAM) d.copy = g.copy_fp4 + static_cast<size_t>(row) * g.ld_copy;
    if (EPI == EPI_STREAM || EPI == EPI_FP4 || EPI == EPI_GEGLU_FP4) d.scales = g.out_scales + scale_offset(row, 0, g.out_blocks);
    return d;
}

// One 32-column chunk of one accumulator row (thread == row); `res` holds the residual of the chunk (BF16) if there is one.
// (Instantiated per epilogue kind: each accumulator drain carries only its own arithmetic and registers.  Values are kept as
// pairs: the packed FP32 operations shorten the straight-line code that a drain executes once.)
// LEAN: without the options only the BF16 model uses (rounding before the residual, GELU on BF16 output) and without ReLU^2.
// TOGETHER: FP32 rows are stored by the whole warp (store_rows64); every lane of the warp calls.
template <int EPI, bool LEAN = false, bool TOGETHER = false>
__device__ __forceinline__ void gemm_epilogue_chunk(const GemmParams& g, const DrainRow& d, const uint32_t (&raw)[32], const uint4 (&res)[4], int row, int col0,
                                                    bool row_ok, float row_scale, float row_shift, float2& sumsq, float2& sum) {
    float2 v[16];
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = mul2(make_float2(__uint_as_float(raw[2 * i]), __uint_as_float(raw[2 * i + 1])), make_float2(row_scale, row_scale));
    constexpr bool kWarpStore = EPI == EPI_BF16 || EPI == EPI_BF16_EXT;      // (rows stored together take the whole warp)
    if (!kWarpStore && !row_ok && !(EPI == EPI_QKV_ROPE && d.together) && !(EPI == EPI_F32 && TOGETHER)) return;
    if constexpr (EPI == EPI_BF16_EXT || EPI == EPI_FP4) {
        if (d.center) {
            // folded LayerNorm: subtract the row mean's share, mean * rstd * (sum over K of weight row n)
            const float4* c4 = reinterpret_cast<const float4*>(d.center + col0);
            const float2 shift = make_float2(row_shift, row_shift);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float4 c = __ldg(c4 + i);
                v[2 * i] = fma2(shift, make_float2(c.x, c.y), v[2 * i]);
                v[2 * i + 1] = fma2(shift, make_float2(c.z, c.w), v[2 * i + 1]);
            }
        }
    }
    if constexpr (EPI == EPI_GEGLU_FP4) {
        // interleaved (gate, up) column pairs -> 16 outputs = one scale block
        float h[16];
#pragma unroll
        for (int i = 0; i < 16; i++) h[i] = gelu_sigmoid(v[i].x) * v[i].y * d.inv_gs;
        uint32_t code;
        uint2 bytes = quantize_block16(h, 0, code);
        const int out_col = col0 >> 1;
        *reinterpret_cast<uint2*>(d.out + (out_col >> 1)) = bytes;
        *scale_at(d, out_col >> 4) = static_cast<uint8_t>(code);
        return;
    }
    if constexpr (EPI == EPI_GEGLU_BF16) {
        // bf16(gelu(bf16 gate)) * bf16(up), rounded once more: the BF16 model's GeGLU on interleaved (gate, up) columns
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float h0 = bf16_round(gelu_tanh(bf16_round(v[2 * i].x))) * bf16_round(v[2 * i].y);
            const float h1 = bf16_round(gelu_tanh(bf16_round(v[2 * i + 1].x))) * bf16_round(v[2 * i + 1].y);
            w[i] = pack_bf16x2(h0, h1);
        }
        uint4* dst = reinterpret_cast<uint4*>(d.out + col0);
        dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
        dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
        return;
    }
    // (residual first, bias second: the order of the reference epilogue, whose BF16 result the tests reproduce bit for bit -
    // but a projection that is rounded before the residual is added carries its bias by then)
    auto add_bias = [&]() {
        const uint4* b = reinterpret_cast<const uint4*>(d.bias + col0 * 2);
        const uint4 u[4] = {__ldg(b), __ldg(b + 1), __ldg(b + 2), __ldg(b + 3)};
        add_bf16x32(v, u);
    };
    const bool early_bias = !LEAN && EPI == EPI_BF16_EXT && d.bias && d.residual && g.round_before_residual;
    if (early_bias) add_bias();
    if (d.residual) {
        if (!LEAN && EPI == EPI_BF16_EXT && g.round_before_residual) {
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = make_float2(bf16_round(v[i].x), bf16_round(v[i].y));
        }
        add_bf16x32(v, res);
    }
    if (d.bias && !early_bias) add_bias();
    if constexpr (EPI == EPI_F32 && TOGETHER) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint4 p[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 a = v[8 * h + 2 * i], b = v[8 * h + 2 * i + 1];
                p[i] = make_uint4(__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(b.x), __float_as_uint(b.y));
            }
            store_rows64(d.out + static_cast<size_t>(col0 + 16 * h) * 4, g.ldo * 4, d.rows_left, p);
        }
        return;
    }
    if constexpr (EPI == EPI_F32) {
        float4* dst = reinterpret_cast<float4*>(d.out + static_cast<size_t>(col0) * 4);
#pragma unroll
        for (int i = 0; i < 8; i++) dst[i] = make_float4(v[2 * i].x, v[2 * i].y, v[2 * i + 1].x, v[2 * i + 1].y);
        return;
    }
    if constexpr (EPI == EPI_STREAM) {
        // the residual stream in BF16 ...
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; i++) w[i] = pack_bf16x2(v[i].x, v[i].y);
        uint4* dst = reinterpret_cast<uint4*>(d.out + col0 * 2);
#pragma unroll
        for (int i = 0; i < 4; i++) dst[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
        // ... and, from the rounded values a norm stage would have read back, the NVFP4 copy and the sums (even and odd
        // columns apart)
#pragma unroll
        for (int i = 0; i < 16; i++) {
            v[i] = unpack_bf16x2(w[i]);
            sumsq = fma2(v[i], v[i], sumsq);
        }
        if (d.sums) {
#pragma unroll
            for (int i = 0; i < 16; i++) sum = add2(sum, v[i]);
        }
        uint32_t codes;
        *reinterpret_cast<uint4*>(d.copy + (col0 >> 1)) = quantize_32(v, d.inv_gs, codes);
        *reinterpret_cast<uint16_t*>(scale_at(d, col0 >> 4)) = static_cast<uint16_t>(codes);
        return;
    }
    if constexpr (EPI == EPI_BF16 || EPI == EPI_BF16_EXT) {
        if (!LEAN && EPI == EPI_BF16_EXT && g.gelu_cols > 0) {
#pragma unroll
            for (int i = 0; i < 16; i++)
                v[i] = make_float2(col0 + 2 * i < g.gelu_cols ? gelu_tanh(bf16_round(v[i].x)) : 0.f,
                                   col0 + 2 * i + 1 < g.gelu_cols ? gelu_tanh(bf16_round(v[i].y)) : 0.f);
        }
        uint4 p[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
            p[i] = make_uint4(pack_bf16x2(v[4 * i].x, v[4 * i].y), pack_bf16x2(v[4 * i + 1].x, v[4 * i + 1].y),
                              pack_bf16x2(v[4 * i + 2].x, v[4 * i + 2].y), pack_bf16x2(v[4 * i + 3].x, v[4 * i + 3].y));
        // padded: heads written pad_to columns apart (8-column pieces never straddle a head: pad_from is a multiple of 8); the
        // lane's piece moves by the gaps in front of it.  Eight rows per store instruction: these drains write wide tiles, whose
        // stores were a third of their time (768 x 32768 BF16 42.0 -> 38.2 us).  In the residual-stream drain, and in q|k|v's of a
        // single row band, the transpose costs more than it saves: few warps are at work there, and the chain of a thread counts
        // (o_proj 5.2 -> 6.1 us).
        const int lane = lane_id();
        int gap = 0;
        if (EPI == EPI_BF16_EXT && g.pad_from > 0) gap = (col0 + (lane & 3) * 8) / g.pad_from * (g.pad_to - g.pad_from);
        store_rows64(d.out + (col0 + gap) * 2, d.ldo, d.rows_left, p);
        return;
    }
    if constexpr (EPI == EPI_FP4) {
        if (d.act == 1) {
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = make_float2(gelu_sigmoid(v[i].x), gelu_sigmoid(v[i].y));
        } else if (!LEAN && d.act == 3) {
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const float2 r = make_float2(fmaxf(v[i].x, 0.f), fmaxf(v[i].y, 0.f));
                v[i] = mul2(r, r);
            }
        }
        uint32_t codes;
        *reinterpret_cast<uint4*>(d.out + (col0 >> 1)) = quantize_32(v, d.inv_gs, codes);
        *reinterpret_cast<uint16_t*>(scale_at(d, col0 >> 4)) = static_cast<uint16_t>(codes);
        return;
    }
    // EPI_QKV_ROPE: values are first rounded to BF16 (the projection output), then rotated.
    if constexpr (EPI == EPI_QKV_ROPE) {
        const int hd = g.head_dim, half = hd >> 1;
        const int kv0 = g.q_cols;                      // K columns [kv0, kv0+hd), V columns [kv0+hd, kv0+2hd)
        const bool is_v = col0 >= kv0 + hd;
        const bool is_k = !is_v && col0 >= kv0;
        const int in_head = is_v ? col0 - kv0 - hd : (is_k ? col0 - kv0 : col0 % hd);
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 16; i++) packed[i] = pack_bf16x2(v[i].x, v[i].y);
        if (!is_v) {
            // Q and K heads are stored pair-interleaved: column 2i holds original dim i, column 2i+1 holds dim i+hd/2; the 16 pairs
            // of this chunk use table entries [dim0, dim0+16) and [dim0+half, dim0+half+16).
            const int dim0 = in_head >> 1;
            // Packed BF16 arithmetic, two lanes = the two members of a rotation pair: with X = (x1, x2), C = (c1, c2),
            // S = (s1, s2) and X' = (-x2, x1) the rotated pair is  bf16(X * C) + bf16(X' * S)  lane by lane - every
            // product rounded to BF16 before the sum, as the reference's rotate-half does.
            auto rotate = [](uint32_t xw, uint32_t cw, uint32_t sw) {      // xw: (x1, x2) rounded to BF16
                const uint32_t xr = __byte_perm(xw, xw, 0x1032u) ^ 0x00008000u;   // (-x2, x1)
                const __nv_bfloat162 p = __hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&xw), *reinterpret_cast<const __nv_bfloat162*>(&cw));
                const __nv_bfloat162 q = __hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&xr), *reinterpret_cast<const __nv_bfloat162*>(&sw));
                const __nv_bfloat162 o = __hadd2_rn(p, q);                  // (_rn: never contracted into a fused multiply-add)
                return *reinterpret_cast<const uint32_t*>(&o);
            };
            if (LEAN || g.rope_table) {
                // the lanes' rows of one pair are adjacent: two lines per load (row by row the eight loads of the two tables take 32
                // lines each, a quarter of the time of a prefix tile)
                const uint2* t = g.rope_table + static_cast<size_t>(dim0) * g.rope_ld + row;
                const int ld = g.rope_ld;
                uint2 cs[16];
#pragma unroll
                for (int i = 0; i < 16; i++) cs[i] = __ldg(t + static_cast<size_t>(i) * ld);
#pragma unroll
                for (int i = 0; i < 16; i++) packed[i] = rotate(packed[i], cs[i].x, cs[i].y);
            } else if constexpr (!LEAN) {
                if (row_ok) {
                    const __nv_bfloat16* cs = static_cast<const __nv_bfloat16*>(g.rope_cos) + static_cast<size_t>(row) * hd;
                    const __nv_bfloat16* sn = static_cast<const __nv_bfloat16*>(g.rope_sin) + static_cast<size_t>(row) * hd;
                    uint32_t tc[2][8], ts[2][8];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint4* pc = reinterpret_cast<const uint4*>(cs + dim0 + h * half);
                        const uint4* ps = reinterpret_cast<const uint4*>(sn + dim0 + h * half);
                        const uint4 c0 = __ldg(pc), c1 = __ldg(pc + 1), s0 = __ldg(ps), s1 = __ldg(ps + 1);
                        tc[h][0] = c0.x; tc[h][1] = c0.y; tc[h][2] = c0.z; tc[h][3] = c0.w;
                        tc[h][4] = c1.x; tc[h][5] = c1.y; tc[h][6] = c1.z; tc[h][7] = c1.w;
                        ts[h][0] = s0.x; ts[h][1] = s0.y; ts[h][2] = s0.z; ts[h][3] = s0.w;
                        ts[h][4] = s1.x; ts[h][5] = s1.y; ts[h][6] = s1.z; ts[h][7] = s1.w;
                    }
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        const uint32_t sel = (i & 1) ? 0x7632u : 0x5410u;      // high or low halves of the two table words
                        packed[i] = rotate(packed[i], __byte_perm(tc[0][i >> 1], tc[1][i >> 1], sel), __byte_perm(ts[0][i >> 1], ts[1][i >> 1], sel));
                    }
                }
            }
        }
        uint8_t* dst;
        int ld = hd * 2;
        if (is_v) dst = static_cast<uint8_t*>(g.cache_v) + (static_cast<size_t>(g.cache_base + row) * hd + in_head) * 2;
        else if (is_k) dst = static_cast<uint8_t*>(g.cache_k) + (static_cast<size_t>(g.cache_base + row) * hd + in_head) * 2;
        else {
            dst = d.out + col0 * 2;
            ld = d.ldo;
        }
        uint4 p[4];
#pragma unroll
        for (int i = 0; i < 4; i++) p[i] = make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
        if (d.together) {
            store_rows64(dst, ld, d.rows_left, p);
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) reinterpret_cast<uint4*>(dst)[i] = p[i];
        }
    }
}

// The drain of one GEMM instruction.  Warps 4 - 7 drain every tile, each the 32 accumulator rows of its tensor-memory
// quarter.  A drain is a serial chain per thread (one row each), 0.5 - 1 us per 32 columns, and behind the last tile of an
// instruction the other warps have nothing left to do: there warp w (0 - 3, same quarter) takes the second half of the
// columns of warp w + 4 ("helped" tiles; not the 32-wide ones, which are a single chunk).  Quarters without logical rows are
// neither drained nor helped.
//
// A helping warp may be an accumulator use or more ahead of the tensor core (copy warps), where the parity of acc_full
// aliases; it therefore does not wait on that barrier but on a word that its partner sets to the ordinal of the GEMM
// instruction once it has seen the accumulator complete.  The partner also leaves the row factors it has computed: the
// helper comes from its role at about that moment and would have to fetch the row statistics first.
// LEAN: the drain of the lean kernel variant; the residual-stream and plain BF16 drains there carry no row-statistics code
// (the host sends programs that give those two epilogues row statistics to the full variant), and that of q|k|v reads the pair-major
// rotary table only.  Of FP32 rows (in the full variants): without bias, residual and row factors kept over tiles, for raw NVFP4 products; with
// them in one drain such products took longer (3 x 8192 x 1024 7.26 us, 6.6 here, 700 x 4352 x 1152 16.6 and 16.2; dense ones did not).
// WIDE: NVFP4 tiles of 192 columns, which take two accumulator uses and may end beyond the logical columns.  An instantiation of its
// own: with both in one drain the others' take 0.1 us longer (one view 5.21 -> 5.31 ms, BF16 16.16 -> 16.51).
template <int EPI, bool LEAN = false, bool WIDE = false>
__device__ __forceinline__ void gemm_epilogue(const VmProgram& prog, Ctl* ctl, uint32_t tmem, const StageDesc& st,
                                              int stage_index, int first, int count, PipeState& ps, long long* stamp) {
    const GemmParams& g = st.p.gemm;
    constexpr bool kStats = !(LEAN && (EPI == EPI_STREAM || EPI == EPI_BF16));
    constexpr bool kResidual = EPI != EPI_GEGLU_FP4 && EPI != EPI_GEGLU_BF16 && EPI != EPI_QKV_ROPE && !(EPI == EPI_F32 && LEAN);
    const int quarter = (threadIdx.x >> 5) & 3;          // TMEM lane quarter this warp may read
    const bool main = threadIdx.x >= 128;
    const int lane = lane_id();
    const int n_tiles = g.n_tiles, block_n = g.block_n, last = first + count - 1;
    constexpr int kUses = WIDE ? 2 : 1;                  // accumulator uses of a tile
    int run = 0;                                         // tiles drained since the last publication
    int known_band = -1;                                 // row band of the tile drained before
    float row_scale = 1.f, row_shift = 0.f;
    for (int t = main ? first : last; t <= last; ++t) {
        const int m_tile = t / n_tiles, n_tile = t - m_tile * n_tiles;
        const uint32_t use = ps.tile + static_cast<uint32_t>((t - first) * kUses);
        const uint32_t buf = use & 1u, phase = (use >> 1) & 1u;
        const int row = m_tile * 128 + quarter * 32 + lane;
        const bool row_ok = row < g.rows;
        const bool rows_here = m_tile * 128 + quarter * 32 < g.rows;
        const bool shared_tile = t == last && block_n >= 64, helped = shared_tile && rows_here;
        if (!main && !helped) break;
        const int col_begin = main ? 0 : block_n >> 1;
        int col_end = main && helped ? block_n >> 1 : block_n;
        if constexpr (WIDE) col_end = min(col_end, g.cols - n_tile * block_n);      // (logical columns are multiples of 32)
        if (EPI == EPI_QKV_ROPE && rows_here) {
            // while the MMAs run: bring the first chunk's rotary table entries (constant data) close
            const int hd = g.head_dim, col_a = n_tile * block_n + col_begin;
            if (col_a < g.q_cols + hd) {                                   // a Q or K tile
                const int in_head = col_a >= g.q_cols ? col_a - g.q_cols : col_a % hd;
                if (LEAN || g.rope_table) {
                    prefetch_l1(g.rope_table + static_cast<size_t>((in_head >> 1) + (lane >> 1)) * g.rope_ld + row - lane + (lane & 1) * 16);
                } else if (!LEAN && row_ok) {
                    const __nv_bfloat16* cs = static_cast<const __nv_bfloat16*>(g.rope_cos) + static_cast<size_t>(row) * hd + (in_head >> 1);
                    const __nv_bfloat16* sn = static_cast<const __nv_bfloat16*>(g.rope_sin) + static_cast<size_t>(row) * hd + (in_head >> 1);
                    prefetch_l1(cs); prefetch_l1(cs + (hd >> 1)); prefetch_l1(sn); prefetch_l1(sn + (hd >> 1));
                }
            }
        }
        if ((EPI == EPI_BF16_EXT || EPI == EPI_FP4) && g.col_center && lane < (block_n >> 5))
            prefetch_l1(g.col_center + n_tile * block_n + lane * 32);    // constant data: close by when the accumulator is ready
        const DrainRow d = drain_row<EPI, LEAN>(g, row);
        // A single-tile instruction that reads row statistics (the few-row projections behind a folded norm, whose epilogue
        // is serial time) or a residual: once the copy warp has seen the sources complete, the statistics are read and the
        // row factor computed, and the first residual chunk is requested, while the operands are still on their way instead
        // of after the accumulator is ready.  (The early residual alone is worth 0.25 of the 10.1 ms pi0 forward.)
        // (compiled into the drains of the projections that stand behind a folded norm in the model; the others read their
        // statistics, if they are given any, once the accumulator is ready)
        constexpr bool kEarly = EPI == EPI_QKV_ROPE || EPI == EPI_GEGLU_FP4 || EPI == EPI_FP4 || EPI == EPI_BF16_EXT;
        const bool early = count == 1 && ((kEarly && (g.row_sumsq != nullptr || g.row_factor != nullptr)) || (kResidual && d.residual != nullptr));
        uint4 res[4] = {};
        auto load_residual = [&](int c) {
            if (kResidual && d.residual && row_ok) {
                const uint4* r = reinterpret_cast<const uint4*>(d.residual + (n_tile * block_n + c) * 2);
#pragma unroll
                for (int i = 0; i < 4; i++) res[i] = __ldcg(r + i);
            }
        };
        volatile float* shared = &ctl->drain_rows[(quarter * 4 + static_cast<int>(ps.gemm_seq & 3u)) * 64 + lane];
        if (!main) {
            if (kResidual && early) {
                if (!word_wait<0>(prog, ctl, &ctl->deps_seen, ps.gemm_seq, stage_index)) return;
                load_residual(col_begin);
            }
            if (!word_wait<0>(prog, ctl, &ctl->drain_seen[quarter], ps.gemm_seq, stage_index)) return;
        } else if (early) {
            if (!word_wait<32>(prog, ctl, &ctl->deps_seen, ps.gemm_seq, stage_index)) return;
            load_residual(0);
        } else {
            if (!mbar_wait_warp(prog, ctl, &ctl->acc_full[buf], phase, stage_index)) return;
        }
        // alpha, times the row's 1/rms where the projection reads un-normalised rows (norm weight folded into B): given
        // as a factor, or as the producer's per-tile sums of squares (complete: the operands behind this accumulator
        // were only copied after the producer stage had finished)
        // (once per row band: a worker's next tiles are mostly of the same one, and the statistics are a round trip to L2)
        const bool factors = (EPI == EPI_F32 && LEAN) || m_tile != known_band;
        known_band = m_tile;
        if (factors) { row_scale = g.alpha; row_shift = 0.f; }
        if (kStats && factors && main && row_ok && g.row_factor) row_scale *= __ldcg(g.row_factor + row);
        if (kStats && factors && main && row_ok && g.row_sumsq) {
            const float4* part = reinterpret_cast<const float4*>(g.row_sumsq + static_cast<size_t>(row) * g.sumsq_parts);
            const int quads = g.sumsq_parts >> 2;
            float total = 0.f;
            if ((EPI == EPI_BF16_EXT || EPI == EPI_FP4) && g.row_sum) {
                // LayerNorm: the per-tile sums (same layout) are requested together with the sums of squares; the mean
                // from the sums, the variance as E[x^2] - mean^2
                const float4* spart = reinterpret_cast<const float4*>(g.row_sum + static_cast<size_t>(row) * g.sumsq_parts);
                float stotal = 0.f;
                for (int i0 = 0; i0 < quads; i0 += 4) {
                    float4 q[4], sq[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        q[j] = i0 + j < quads ? __ldcg(part + i0 + j) : make_float4(0.f, 0.f, 0.f, 0.f);
                        sq[j] = i0 + j < quads ? __ldcg(spart + i0 + j) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) {                    // fixed order: the same bits on every launch
                        if (i0 + j < quads) {
                            total += q[j].x; total += q[j].y; total += q[j].z; total += q[j].w;
                            stotal += sq[j].x; stotal += sq[j].y; stotal += sq[j].z; stotal += sq[j].w;
                        }
                    }
                }
                const float mean = stotal * g.sumsq_inv_width;
                const float rstd = rsqrtf(fmaxf(total * g.sumsq_inv_width - mean * mean, 0.f) + g.sumsq_eps);
                row_scale *= rstd;
                row_shift = -mean * rstd;
            } else {
                for (int i0 = 0; i0 < quads; i0 += 8) {              // eight loads in flight: one L2 round trip per 128 bytes
                    float4 q[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) q[j] = i0 + j < quads ? __ldcg(part + i0 + j) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int j = 0; j < 8; j++) {                    // fixed order: the same bits on every launch
                        if (i0 + j < quads) { total += q[j].x; total += q[j].y; total += q[j].z; total += q[j].w; }
                    }
                }
                row_scale *= rsqrtf(total * g.sumsq_inv_width + g.sumsq_eps);
            }
        }
        if (main) {
            if (early && !mbar_wait_warp(prog, ctl, &ctl->acc_full[buf], phase, stage_index)) return;
            if (helped) {
                if (kStats) { shared[0] = row_scale; shared[32] = row_shift; }
                __syncwarp();
                if (lane == 0) word_set(&ctl->drain_seen[quarter], ps.gemm_seq + 1u);
            }
        } else if (kStats) {
            row_scale = shared[0];
            row_shift = shared[32];
        }
        tc_fence_after();
        if (stamp && t == first && threadIdx.x == 128) stamp[6] = static_cast<long long>(global_ns());
        const uint32_t taddr = tmem + (WIDE ? 0u : buf * 128u) + (static_cast<uint32_t>(quarter * 32) << 16);
        const uint32_t share = helped ? 1u : 2u;             // parts of the tile this warp speaks for: two per quarter
        auto columns_read = [&]() {                          // this warp's part of the accumulator is in registers
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_count(&ctl->acc_empty[buf], share);
            if (WIDE && lane == 0) mbar_arrive_count(&ctl->acc_empty[buf ^ 1u], share);
        };
        // Residual-stream statistics: the two halves of a tile are summed apart, whichever warps drain them, and added at the
        // end, so the bits do not depend on how the tiles are dealt to the workers.
        float2 sumsq = make_float2(0.f, 0.f), sum = make_float2(0.f, 0.f);
        float sumsq_half = 0.f, sum_half = 0.f;
        if (!rows_here || (WIDE && col_begin >= col_end)) {
            columns_read();
        } else {
            if (!early) load_residual(col_begin);
#pragma unroll 1
            for (int c = col_begin; c < col_end; c += 32) {
                uint32_t raw[32];
                tmem_ld32(taddr + c, raw);
                tmem_ld_wait();
                if (c + 32 == col_end) columns_read();
                if (EPI == EPI_STREAM && main && block_n >= 64 && c == block_n >> 1) {
                    sumsq_half = sumsq.x + sumsq.y;
                    sum_half = sum.x + sum.y;
                    sumsq = sum = make_float2(0.f, 0.f);
                }
                gemm_epilogue_chunk<EPI, LEAN>(g, d, raw, res, row, n_tile * block_n + c, row_ok, row_scale, row_shift, sumsq, sum);
                if (c + 32 < col_end) load_residual(c + 32);
            }
        }
        if (EPI == EPI_STREAM && rows_here) {
            float a = sumsq.x + sumsq.y, b = sum.x + sum.y;
            if (!main) {                                     // second half: handed to the partner
                shared[0] = a;
                shared[32] = b;
                __syncwarp();
                if (lane == 0) word_set(&ctl->sums_seen[quarter], ps.gemm_seq + 1u);
            } else {
                if (helped) {
                    if (!word_wait<0>(prog, ctl, &ctl->sums_seen[quarter], ps.gemm_seq, stage_index)) return;
                    sumsq_half = shared[0];
                    sum_half = shared[32];
                }
                if (row_ok) {
                    g.sumsq_out[static_cast<size_t>(row) * g.sumsq_ld + n_tile] = a + sumsq_half;
                    if (g.sum_out) g.sum_out[static_cast<size_t>(row) * g.sumsq_ld + n_tile] = b + sum_half;
                }
            }
        }
        // The tiles of a run - one row band, one instruction - are published together and once, by whichever warp finishes
        // last.  A counter that takes one increment per warp of every tile serialises them in L2 (40 tiles x 6 warps: the
        // attention behind q|k|v saw its sources 0.6 us later), and the fences in front of it wait for the stores.
        run++;
        if (t != last && (t + 1) / n_tiles == m_tile) continue;
        if (stamp && t == last && threadIdx.x == 128) stamp[7] = static_cast<long long>(global_ns());
        fence_proxy_async_global();
        __syncwarp();
        if (lane == 0 && join_parts(&ctl->tile_parts[shared_tile ? 4u + (ps.gemm_seq & 3u) : ps.run & 3u], share))
            publish_tile(prog, st, t, static_cast<unsigned int>(main ? run : min(count, t - m_tile * n_tiles + 1)));
        run = 0;
        if (!shared_tile) ps.run++;
    }
    ps.tile += static_cast<uint32_t>(count * kUses);
}

// Dispatch of one GEMM instruction onto the warp roles (warp 2 has none); behind its role every warp goes through the
// drain, as one of the draining warps or as a helper of the last tile.
// LEAN: the kernel variant for programs made only of NVFP4 projections with the pi0 model's epilogues (the host checks
// this when it builds a program); it carries neither the dense issue loops nor the other drain loops.
// WIDE: with the forms for 192-wide NVFP4 tiles.  ROTARY_ROWS: with those for rotary tables row by row.
template <bool LEAN, bool WIDE, bool ROTARY_ROWS>
__device__ __forceinline__ void gemm_instruction(const VmProgram& prog, Ctl* ctl, uint8_t* data, uint32_t tmem,
                                                 const StageDesc& st, int stage_index, int first, int count,
                                                 PipeState& ps, long long* stamp) {
    const int warp = threadIdx.x >> 5;
    if (warp == 0) {
        gemm_producer<false, WIDE || !LEAN>(prog, ctl, data, st, stage_index, first, count, ps, stamp);
        if (stamp && threadIdx.x == 0) stamp[3] = static_cast<long long>(global_ns());
    } else if (warp == 3) {
        gemm_producer<true, WIDE || !LEAN>(prog, ctl, data, st, stage_index, first, count, ps, nullptr);
    } else if (warp == 1) {
        const int operands = st.p.gemm.operands;
        if (LEAN || operands == GEMM_NVFP4) gemm_mma<GEMM_NVFP4, WIDE>(prog, ctl, data, tmem, st, stage_index, first, count, ps, stamp);
        else if (operands == GEMM_BF16) gemm_mma<GEMM_BF16, false>(prog, ctl, data, tmem, st, stage_index, first, count, ps, stamp);
        else gemm_mma<GEMM_FP8, false>(prog, ctl, data, tmem, st, stage_index, first, count, ps, stamp);
    }
    const int epilogue = st.p.gemm.epilogue;                // one drain loop per epilogue kind: only its own arithmetic and registers
    if (WIDE && __builtin_expect(st.p.gemm.block_n > 128, 0)) {
        if (epilogue == EPI_FP4) gemm_epilogue<EPI_FP4, LEAN, WIDE>(prog, ctl, tmem, st, stage_index, first, count, ps, stamp);
        else gemm_epilogue<EPI_BF16_EXT, LEAN, WIDE>(prog, ctl, tmem, st, stage_index, first, count, ps, stamp);
    } else if (epilogue == EPI_BF16) gemm_epilogue<EPI_BF16, LEAN>(prog, ctl, tmem, st, stage_index, first, count, ps, stamp);
    else if (epilogue == EPI_STREAM) gemm_epilogue<EPI_STREAM, LEAN>(prog, ctl, tmem, st, stage_index, first, count, ps, stamp);
    else if (epilogue == EPI_GEGLU_FP4) gemm_epilogue<EPI_GEGLU_FP4, LEAN>(prog, ctl, tmem, st, stage_index, first, count, ps, stamp);
    else if (epilogue == EPI_FP4) gemm_epilogue<EPI_FP4, LEAN>(prog, ctl, tmem, st, stage_index, first, count, ps, stamp);
    else if (epilogue == EPI_QKV_ROPE) gemm_epilogue<EPI_QKV_ROPE, LEAN && !ROTARY_ROWS>(prog, ctl, tmem, st, stage_index, first, count, ps, stamp);
    else if (LEAN || epilogue == EPI_BF16_EXT) gemm_epilogue<EPI_BF16_EXT, LEAN>(prog, ctl, tmem, st, stage_index, first, count, ps, stamp);
    else if (epilogue == EPI_F32 && st.p.gemm.operands == GEMM_NVFP4 && !st.p.gemm.bias && !st.p.gemm.residual)
        gemm_epilogue<EPI_F32, true>(prog, ctl, tmem, st, stage_index, first, count, ps, stamp);
    else if (epilogue == EPI_F32) gemm_epilogue<EPI_F32>(prog, ctl, tmem, st, stage_index, first, count, ps, stamp);
    else gemm_epilogue<EPI_GEGLU_BF16>(prog, ctl, tmem, st, stage_index, first, count, ps, stamp);
    if (stamp && threadIdx.x == 128) stamp[2] = static_cast<long long>(global_ns());
    ps.gemm_seq++;                                          // (every warp: the ordinal of the next GEMM instruction of this CTA)
}

}  // namespace pi0
