// Small FP32 operators around the transformer blocks: patch embedding, token embedding, FP32 linears with fused
// SiLU / RMS factor / Euler update, and the expert-input assembly. All are CTA-wide, coalesced CUDA-core code.
#pragma once
#include "vm_core.cuh"
#include "op_norm.cuh"
#include "op_attention.cuh"

namespace pi0 {

// Patch embedding: out[t, n] = sum_k patch[t, k] * W[k, n] + bias[n] + pos[t % 256, n];  k = (dy*14 + dx)*3 + c, images are NHWC.
//
// 1 GFLOP in FP32 for three views, and the first stage of the model: nothing else runs beside it.  A tile is 16 tokens (8 when
// there is only one view, for twice the CTAs) by 384 columns, which gives 144 tiles for the three views of pi0 - one wave.
// A warp serves 32 columns, 32 + 128 and 32 + 256 for one half of the tokens, so a k costs two broadcast reads of patch
// values (stored [k][token]), three of weights and twelve packed multiply-adds; the weights come through a six-deep
// cp.async ring of 14 k each.  (One column per thread with the weights read straight from L2 was bound by the latency of
// those reads: 157 us for three views, 103 for one.)
constexpr int kPatchCols = 384;
constexpr int kPatchK = 14 * 14 * 3;                                   // 588
constexpr int kPatchStageK = 14;
constexpr int kPatchStages = 6;
constexpr int kPatchStageBytes = kPatchStageK * kPatchCols * 4;
constexpr int kPatchLd = 20;                                           // floats per k of patch values (16 tokens, padded)
static_assert(kPatchK % kPatchStageK == 0 && kPatchK * kPatchLd * 4 + kPatchStages * kPatchStageBytes <= kDataBytes, "patch tile exceeds the data region");

__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool valid) {
    const int bytes = valid ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void patch_issue(const PatchParams& p, float* stage, int k0, int n0) {
    const float* w = p.weight + static_cast<size_t>(k0) * p.width + n0;
    if ((p.width & 3) == 0 && (reinterpret_cast<uintptr_t>(p.weight) & 15u) == 0) {
        for (int i = threadIdx.x; i < kPatchStageK * (kPatchCols / 4); i += kThreads) {
            const int r = i / (kPatchCols / 4), c = (i - r * (kPatchCols / 4)) * 4;
            const bool ok = n0 + c < p.width;
            cp_async16(stage + r * kPatchCols + c, ok ? w + static_cast<size_t>(r) * p.width + c : p.weight, ok);
        }
    } else {
        for (int i = threadIdx.x; i < kPatchStageK * kPatchCols; i += kThreads) {
            const int r = i / kPatchCols, c = i - r * kPatchCols;
            const bool ok = n0 + c < p.width;
            cp_async4(stage + i, ok ? w + static_cast<size_t>(r) * p.width + c : p.weight, ok);
        }
    }
}
template <int TOKENS>
__device__ __forceinline__ void patch_tile(const PatchParams& p, const float* images, int tile, uint8_t* data) {
    constexpr int kHalf = TOKENS / 2, kPairs = TOKENS / 4;             // tokens / token pairs of one thread
    float* sp = reinterpret_cast<float*>(data);                        // [588][kPatchLd]
    float* ring = sp + kPatchK * kPatchLd;                             // [stages][14][384]
    const int ntiles = (p.width + kPatchCols - 1) / kPatchCols;
    const int tt = tile / ntiles, n0 = (tile - tt * ntiles) * kPatchCols;
    for (int s = 0; s < kPatchStages - 1; ++s) {
        patch_issue(p, ring + s * (kPatchStageBytes / 4), s * kPatchStageK, n0);
        cp_async_commit();
    }
    // gather the patches: loads are issued in batches of 8 per thread before any is stored
    for (int base = 0; base < TOKENS * kPatchK; base += kThreads * 8) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int i = base + j * kThreads + threadIdx.x;
            v[j] = 0.f;
            if (i < TOKENS * kPatchK) {
                const int tok = i / kPatchK, k = i - tok * kPatchK;
                const int dy = k / 42, rem = k - dy * 42;
                const int t = tt * TOKENS + tok;
                const int view = t >> 8, pidx = t & 255, py = pidx >> 4, px = pidx & 15;
                v[j] = __ldg(images + ((static_cast<size_t>(view) * 224 + py * 14 + dy) * 224 + px * 14) * 3 + rem);
            }
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int i = base + j * kThreads + threadIdx.x;
            if (i < TOKENS * kPatchK) {
                const int tok = i / kPatchK;
                sp[(i - tok * kPatchK) * kPatchLd + tok] = v[j];
            }
        }
    }
    const int half = threadIdx.x >> 7, col = threadIdx.x & 127;
    float2 acc[3][kPairs];
#pragma unroll
    for (int j = 0; j < 3; j++)
#pragma unroll
        for (int i = 0; i < kPairs; i++) acc[j][i] = make_float2(0.f, 0.f);
    constexpr int kSteps = kPatchK / kPatchStageK;
    for (int s = 0; s < kSteps; ++s) {
        cp_async_wait<kPatchStages - 2>();
        __syncthreads();                                               // the stage (and, first, the patches) of every thread; stage s - 1 is free
        const int next = s + kPatchStages - 1;
        if (next < kSteps) patch_issue(p, ring + (next % kPatchStages) * (kPatchStageBytes / 4), next * kPatchStageK, n0);
        cp_async_commit();
        const float* w = ring + (s % kPatchStages) * (kPatchStageBytes / 4) + col;
        const float* x = sp + s * kPatchStageK * kPatchLd + half * kHalf;
#pragma unroll 2
        for (int k = 0; k < kPatchStageK; ++k) {
            float2 xp[kPairs];
#pragma unroll
            for (int i = 0; i < kPairs; i += 2) {
                const float4 q = *reinterpret_cast<const float4*>(x + k * kPatchLd + 2 * i);
                xp[i] = make_float2(q.x, q.y);
                xp[i + 1] = make_float2(q.z, q.w);
            }
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const float wk = w[k * kPatchCols + 128 * j];
#pragma unroll
                for (int i = 0; i < kPairs; i++) acc[j][i] = fma2(xp[i], make_float2(wk, wk), acc[j][i]);
            }
        }
    }
    cp_async_wait<0>();
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const int n = n0 + col + 128 * j;
        if (n < p.width) {
            // (the position rows are read before the first store: the compiler cannot know that they do not overlap the output,
            // and a load behind every store would be a chain of round trips)
            const int t0 = tt * TOKENS + half * kHalf;
            const float b = __ldg(p.bias + n);
            float pos[kHalf];
#pragma unroll
            for (int i = 0; i < kHalf; i++) pos[i] = __ldg(p.pos + static_cast<size_t>((t0 + i) & 255) * p.width + n);
#pragma unroll
            for (int i = 0; i < kHalf; i++) {
                const float y = (i & 1 ? acc[j][i >> 1].y : acc[j][i >> 1].x) + b + pos[i];
                static_cast<__nv_bfloat16*>(p.out)[static_cast<size_t>(t0 + i) * p.width + n] = __float2bfloat16_rn(y);
            }
        }
    }
}

__device__ __forceinline__ void patch_instruction(const VmProgram& prog, Ctl* ctl, uint8_t* data, const StageDesc& st,
                                                  int stage_index, int first, int count) {
    const PatchParams& p = st.p.patch;
    const float* images = p.images ? p.images : prog.in.images;
    for (int t = first; t < first + count; ++t) {
        if (p.tokens == 16) patch_tile<16>(p, images, t, data);
        else patch_tile<8>(p, images, t, data);
        cta_publish_tile(prog, st, t);                                 // (its barrier also frees the buffers for the next tile)
    }
}

// Token rows: out[row_base + i, :] = bf16(table[token_i, :] * scale); eight tokens per tile, one warp each.
__device__ __forceinline__ void embed_instruction(const VmProgram& prog, Ctl* ctl, const StageDesc& st, int stage_index,
                                                  int first, int count) {
    const EmbedParams& e = st.p.embed;
    const long long* tokens = e.tokens ? e.tokens : prog.in.tokens;
    const int warp = threadIdx.x >> 5, lane = lane_id();
    for (int t = first; t < first + count; ++t) {
        const int i = t * 8 + warp;
        if (i < e.count) {
            long long tok = tokens[i];
            tok = tok < 0 ? 0 : (tok >= e.vocab ? e.vocab - 1 : tok);
            const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(e.table) + static_cast<size_t>(tok) * e.width;
            __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(e.out) + static_cast<size_t>(e.row_base + i) * e.width;
            if (e.width % 8 == 0 && ((reinterpret_cast<uintptr_t>(e.table) | reinterpret_cast<uintptr_t>(e.out)) & 15u) == 0) {
                // 16 bytes per lane and load, eight loads in flight (element by element the row was a chain of 64 round trips:
                // 32 us for a prompt)
                const int pieces = e.width >> 3;
                for (int c0 = lane; c0 < pieces; c0 += 256) {
                    uint4 u[8];
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        if (c0 + 32 * j < pieces) u[j] = __ldg(reinterpret_cast<const uint4*>(src) + c0 + 32 * j);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        if (c0 + 32 * j >= pieces) break;
                        const uint32_t in[4] = {u[j].x, u[j].y, u[j].z, u[j].w};
                        uint32_t w[4];
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&in[q]));
                            w[q] = pack2_bf16(f.x * e.scale, f.y * e.scale);
                        }
                        reinterpret_cast<uint4*>(dst)[c0 + 32 * j] = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            } else {
                for (int c = lane; c < e.width; c += 32) dst[c] = __float2bfloat16_rn(__bfloat162float(src[c]) * e.scale);
            }
        }
        cta_publish_tile(prog, st, t);
    }
}

// out[r, n] = f(sum_k x[r, k] * W[n, k]) in FP32.  A tile is 16 output columns for a block of 32 rows (16 for an operator
// with few rows or few columns, which would otherwise occupy one or two CTAs). K runs in chunks of 256 through a four-deep
// cp.async ring in shared memory (x rows as stored, FP32 or BF16, and the 16 weight rows), so the L2 latency of a
// chunk is paid once per tile, not once per chunk.
//
// With eight warps per SM the operator is bound by instruction issue, so the inner loop is built for few instructions:
// every warp owns one eighth of each K chunk (32 values) and computes the WHOLE tile for it - lane (rg = lane / 4,
// cg = lane % 4) holds rows rg, rg + 8, ... and columns cg, cg + 4, cg + 8, cg + 12 - with packed FP32 multiply-adds
// (fma.rn.f32x2: two products per instruction, accumulated as separate even / odd partial sums).  A step of four k
// values costs RT + 4 16-byte shared-memory reads (conflict-free: rows are 132 floats apart) for 8 RT packed
// multiply-adds.  The eight partial tiles meet in shared memory at the end and are added in a fixed order.
constexpr int kLinCols = 16;
constexpr int kLinRows = 32;
constexpr int kLinChunk = 256;
constexpr int kLinLd = kLinChunk + 4;                                  // floats per staged row (padded)
constexpr int kLinStages = 4;
constexpr int kLinStageBytes = (kLinRows + kLinCols) * kLinLd * 4;     // x block + weight rows
static_assert(kLinStages * kLinStageBytes <= kDataBytes, "linear32 ring exceeds the data region");
static_assert(8 * (kLinRows * kLinCols + kLinRows) * 4 <= kLinStages * kLinStageBytes, "partial sums exceed the ring");

// Geometry of one tile, read once from the (shared-memory) descriptor.
struct LinTile {
    const void* x;
    const float* w;
    int rows, n, k, ldx, x_row_offset, x_bf16;
    int col0, r0;
};

// One K chunk into a ring stage: warp w copies rows w, w + 8, ...; lane l the l-th 16-byte piece of the row.
__device__ __forceinline__ void linear32_issue_x(const LinTile& t, uint8_t* stage, int row_block, int kc) {
    const int warp = threadIdx.x >> 5, lane = lane_id();
    const int kw = min(kLinChunk, t.k - kc);
    float* xs = reinterpret_cast<float*>(stage);
    if (t.x_bf16) {
        // BF16 rows are staged as stored (8 elements per 16-byte copy) in the first half of each padded row
        const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(t.x);
        for (int c = lane; c < (kw >> 3); c += 32)
            for (int r = warp; r < row_block; r += 8) {
                const bool ok = t.r0 + r < t.rows;
                const __nv_bfloat16* from = ok ? src + static_cast<size_t>(t.r0 + r + t.x_row_offset) * t.ldx + kc + c * 8 : src;
                cp_async16(reinterpret_cast<__nv_bfloat16*>(xs + r * kLinLd) + c * 8, from, ok);
            }
    } else {
        const float* src = static_cast<const float*>(t.x);
        for (int c = lane; c < (kw >> 2); c += 32)
            for (int r = warp; r < row_block; r += 8) {
                const bool ok = t.r0 + r < t.rows;
                const float* from = ok ? src + static_cast<size_t>(t.r0 + r + t.x_row_offset) * t.ldx + kc + c * 4 : src;
                cp_async16(xs + r * kLinLd + c * 4, from, ok);
            }
    }
}
__device__ __forceinline__ void linear32_issue_w(const LinTile& t, uint8_t* stage, int kc) {
    const int warp = threadIdx.x >> 5, lane = lane_id();
    const int kw = min(kLinChunk, t.k - kc);
    float* ws = reinterpret_cast<float*>(stage) + kLinRows * kLinLd;
    for (int c = lane; c < (kw >> 2); c += 32)
        for (int r = warp; r < kLinCols; r += 8) {
            const bool ok = t.col0 + r < t.n;
            const float* from = ok ? t.w + static_cast<size_t>(t.col0 + r) * t.k + kc + c * 4 : t.w;
            cp_async16(ws + r * kLinLd + c * 4, from, ok);
        }
}

// `wait` (first tile of an instruction): waits for the sources.  Weights do not depend on them, so those of the first
// kLinStages chunks are requested before (Euler update of 51 rows inside the model 14.0 -> 10.9 us).
// FORM: 0 FP32 rows without the RMS factor, 1 BF16 rows with it - the two the model runs, with nothing else in their inner
// loops, which have to fit the instruction buffer of a scheduler - and 2 any combination.
template <int RT, int FORM, typename Wait>
__device__ __forceinline__ bool linear32_tile(const Linear32Params& p, const void* xbase, const float* prev, int tile,
                                              uint8_t* data, bool waits, Wait wait, long long* stamp) {
    constexpr int row_block = 8 * RT;
    const int col_tiles = (p.n + kLinCols - 1) / kLinCols;
    LinTile t;
    t.x = xbase; t.w = p.w;
    t.rows = p.rows; t.n = p.n; t.k = p.k; t.ldx = p.ldx; t.x_row_offset = p.x_row_offset; t.x_bf16 = p.x_bf16;
    t.col0 = (tile % col_tiles) * kLinCols;
    t.r0 = (tile / col_tiles) * row_block;
    const int warp = threadIdx.x >> 5, lane = lane_id();
    const int rg = lane >> 2, cg = lane & 3;
    const int nchunks = (t.k + kLinChunk - 1) / kLinChunk;
    const bool rms = FORM == 2 ? p.rms != 0 : FORM == 1, x_bf16 = FORM == 2 ? t.x_bf16 != 0 : FORM == 1;
    float2 acc[RT][4], ss[RT];
#pragma unroll
    for (int i = 0; i < RT; i++) {
        ss[i] = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = make_float2(0.f, 0.f);
    }
    __syncthreads();                                   // the previous tile's readers are done with the ring
    for (int s = 0; s < kLinStages; ++s)
        if (s < nchunks) linear32_issue_w(t, data + s * kLinStageBytes, s * kLinChunk);
    cp_async_commit();
    if (waits && !wait()) return false;
    for (int s = 0; s < kLinStages - 1; ++s) {
        if (s < nchunks) linear32_issue_x(t, data + s * kLinStageBytes, row_block, s * kLinChunk);
        cp_async_commit();
    }
#pragma unroll 1
    for (int c = 0; c < nchunks; ++c) {
        cp_async_wait<kLinStages - 2>();           // chunk c has landed (this thread's copies) ...
        __syncthreads();                           // ... and everybody's; the buffer of chunk c - 1 is free
        if (stamp && c == 0 && threadIdx.x == 0) stamp[4] = static_cast<long long>(global_ns());
        const int next = c + kLinStages - 1;
        if (next < nchunks) {
            linear32_issue_x(t, data + (next % kLinStages) * kLinStageBytes, row_block, next * kLinChunk);
            if (next >= kLinStages) linear32_issue_w(t, data + (next % kLinStages) * kLinStageBytes, next * kLinChunk);
        }
        cp_async_commit();
        const float* xs = reinterpret_cast<const float*>(data + (c % kLinStages) * kLinStageBytes);
        const float* ws = xs + kLinRows * kLinLd;
        const int kw4 = min(kLinChunk, t.k - c * kLinChunk) >> 2;
#pragma unroll 1
        for (int j = 0; j < kLinChunk / 32; j++) {     // (not unrolled: the operator runs a few times per pass, from a cold instruction cache)
            const int q = warp * (kLinChunk / 32) + j; // this warp's share of the chunk: k values 32 warp .. 32 warp + 31
            if (q < kw4) {
                float4 w4[4];
#pragma unroll
                for (int cc = 0; cc < 4; cc++) w4[cc] = *reinterpret_cast<const float4*>(ws + (cg + 4 * cc) * kLinLd + q * 4);
                constexpr int XB = RT < 4 ? RT : 4;    // rows in flight at a time (register budget)
#pragma unroll
                for (int i0 = 0; i0 < RT; i0 += XB) {
                    float4 x4[XB];
#pragma unroll
                    for (int i = 0; i < XB; i++) {
                        if (x_bf16) {
                            const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(xs + (rg + 8 * (i0 + i)) * kLinLd) + q * 4);
                            const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
                            const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
                            x4[i] = make_float4(lo.x, lo.y, hi.x, hi.y);
                        } else {
                            x4[i] = *reinterpret_cast<const float4*>(xs + (rg + 8 * (i0 + i)) * kLinLd + q * 4);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < XB; i++) {
                        const float2 xa = make_float2(x4[i].x, x4[i].y), xb = make_float2(x4[i].z, x4[i].w);
#pragma unroll
                        for (int cc = 0; cc < 4; cc++)
                            acc[i0 + i][cc] = fma2(xb, make_float2(w4[cc].z, w4[cc].w), fma2(xa, make_float2(w4[cc].x, w4[cc].y), acc[i0 + i][cc]));
                        if (rms) ss[i0 + i] = fma2(xb, xb, fma2(xa, xa, ss[i0 + i]));
                    }
                }
            }
        }
    }
    cp_async_wait<0>();
    __syncthreads();                                   // the ring is free: it now holds the partial sums
    if (stamp && threadIdx.x == 0) stamp[5] = static_cast<long long>(global_ns());
    float* red = reinterpret_cast<float*>(data);       // [8 warps][row_block][16 columns]
    float* red_ss = red + 8 * row_block * kLinCols;    // [8 warps][row_block]
#pragma unroll
    for (int i = 0; i < RT; i++) {
#pragma unroll
        for (int cc = 0; cc < 4; cc++) red[(warp * row_block + rg + 8 * i) * kLinCols + cg + 4 * cc] = acc[i][cc].x + acc[i][cc].y;
        if (cg == 0) red_ss[warp * row_block + rg + 8 * i] = ss[i].x + ss[i].y;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < row_block * kLinCols; o += kThreads) {
        const int rl = o >> 4, cl = o & 15;
        const int r = t.r0 + rl, n = t.col0 + cl;
        if (r >= t.rows || n >= t.n) continue;
        float v = 0.f, sq = 0.f;
#pragma unroll
        for (int k8 = 0; k8 < 8; k8++) {
            v += red[(k8 * row_block + rl) * kLinCols + cl];
            sq += red_ss[k8 * row_block + rl];
        }
        if (rms) v *= rsqrtf(sq / static_cast<float>(t.k) + p.eps);
        if (p.bias) v += p.bias[n];
        if (p.silu) v = v / (1.f + expf(-v));
        if (p.euler) v = __fadd_rn(__ldcg(prev + static_cast<size_t>(r) * t.n + n), __fmul_rn(p.dt, v));
        if (p.out_bf16) static_cast<__nv_bfloat16*>(p.out)[static_cast<size_t>(r) * p.ldo + n] = __float2bfloat16_rn(v);
        else static_cast<float*>(p.out)[static_cast<size_t>(r) * p.ldo + n] = v;
    }
    if (stamp && threadIdx.x == 0) stamp[6] = static_cast<long long>(global_ns());
    // Optional extra row: FP32 values of this tile's columns copied (as BF16) to the row in front of the output,
    // which is how the state token joins the action tokens without a stage of its own.
    if (p.row0_src && t.r0 == 0 && threadIdx.x < kLinCols && t.col0 + threadIdx.x < t.n)
        static_cast<__nv_bfloat16*>(p.row0_dst)[t.col0 + threadIdx.x] = __float2bfloat16_rn(__ldcg(p.row0_src + t.col0 + threadIdx.x));
    return true;
}

// LEAN: the forms of the lean kernel variant (lean_stage).
template <bool LEAN>
__device__ __forceinline__ void linear32_instruction(const VmProgram& prog, Ctl* ctl, uint8_t* data, const StageDesc& st,
                                                     int stage_index, int first, int count, long long* stamp) {
    const Linear32Params& p = st.p.lin;
    const void* xbase = p.slot == 2 ? static_cast<const void*>(prog.in.state)
                        : p.slot == 3 ? static_cast<const void*>(prog.in.noise) : p.x;
    const float* prev = p.prev_slot == 3 ? prog.in.noise : p.prev;
    for (int t = first; t < first + count; ++t) {
        long long* stamp_t = t == first ? stamp : nullptr;
        auto wait = [&]() { return cta_wait_sources(prog, ctl, st, stage_index, first, count, stamp); };
        const int form = p.x_bf16 && p.rms ? 1 : p.x_bf16 || p.rms ? 2 : 0;
        bool ok = false;
        if (p.row_block == 16) {
            if (form == 0) ok = linear32_tile<2, 0>(p, xbase, prev, t, data, t == first, wait, stamp_t);
            else if (LEAN || form == 1) ok = linear32_tile<2, 1>(p, xbase, prev, t, data, t == first, wait, stamp_t);
            else if constexpr (!LEAN) ok = linear32_tile<2, 2>(p, xbase, prev, t, data, t == first, wait, stamp_t);
        } else {
            if (LEAN || form == 0) ok = linear32_tile<4, 0>(p, xbase, prev, t, data, t == first, wait, stamp_t);
            else if constexpr (!LEAN) ok = linear32_tile<4, 2>(p, xbase, prev, t, data, t == first, wait, stamp_t);
        }
        if (!ok) return;                               // uniform: the abort flag is set, the caller leaves the loop
        cta_publish_tile(prog, st, t);
    }
}

// Expert input: row 0 = state embedding, rows 1..chunk = action/time embeddings, as BF16. Eight rows per tile.
__device__ __forceinline__ void suffix_instruction(const VmProgram& prog, Ctl* ctl, const StageDesc& st, int stage_index,
                                                   int first, int count) {
    const SuffixParams& p = st.p.suffix;
    const int warp = threadIdx.x >> 5, lane = lane_id();
    for (int t = first; t < first + count; ++t) {
        const int r = t * 8 + warp;
        if (r <= p.chunk) {
            const float* src = r == 0 ? p.state_emb : p.action_emb + static_cast<size_t>(r - 1) * p.width;
            __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(p.out) + static_cast<size_t>(r) * p.width;
            for (int c = lane; c < p.width; c += 32) dst[c] = __float2bfloat16_rn(__ldcg(src + c));
        }
        cta_publish_tile(prog, st, t);
    }
}

// Attention operand preparation: a tile is eight rows (a warp each) of the concatenated row space Q | K | V.
constexpr int kPrepRows = 8;
__device__ __forceinline__ int prep_tiles(const PrepParams& p) {
    return (p.rows[0] + kPrepRows - 1) / kPrepRows + (p.rows[1] + kPrepRows - 1) / kPrepRows + (p.rows[2] + kPrepRows - 1) / kPrepRows;
}
__device__ __forceinline__ void prep_instruction(const VmProgram& prog, Ctl* ctl, const StageDesc& st, int first, int count) {
    const PrepParams& p = st.p.prep;
    const int warp = threadIdx.x >> 5, lane = lane_id();
    const int tq = (p.rows[0] + kPrepRows - 1) / kPrepRows, tk = (p.rows[1] + kPrepRows - 1) / kPrepRows;
    const int half = p.head_dim >> 1;
    for (int t = first; t < first + count; ++t) {
        const int part = t < tq ? 0 : (t < tq + tk ? 1 : 2);
        const int row = (t - (part == 0 ? 0 : part == 1 ? tq : tq + tk)) * kPrepRows + warp;
        if (row < p.rows[part]) {
            const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(p.src[part]) + static_cast<size_t>(row) * p.ld_src[part];
            __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(p.dst[part]) + static_cast<size_t>(row) * p.ld_dst[part];
            const __nv_bfloat16* bias = static_cast<const __nv_bfloat16*>(p.bias[part]);
            const __nv_bfloat16* cs = part < 2 && p.cos[part] ? static_cast<const __nv_bfloat16*>(p.cos[part]) + static_cast<size_t>(row) * p.head_dim : nullptr;
            const __nv_bfloat16* sn = part < 2 && p.sin[part] ? static_cast<const __nv_bfloat16*>(p.sin[part]) + static_cast<size_t>(row) * p.head_dim : nullptr;
            for (int i = lane; i < p.heads[part] * half; i += 32) {
                const int h = i / half, d = i - h * half;
                float lo = __bfloat162float(src[h * p.src_pitch + d]), hi = __bfloat162float(src[h * p.src_pitch + half + d]);
                if (bias) {
                    lo += __bfloat162float(bias[h * p.head_dim + d]);
                    hi += __bfloat162float(bias[h * p.head_dim + half + d]);
                }
                if (cs) {
                    const float c = __bfloat162float(cs[d]), s = __bfloat162float(sn[d]);
                    const float rl = lo * c - hi * s, rh = hi * c + lo * s;
                    lo = rl; hi = rh;
                }
                dst[h * p.pitch + d] = __float2bfloat16_rn(lo);
                dst[h * p.pitch + half + d] = __float2bfloat16_rn(hi);
            }
        }
        cta_publish_tile(prog, st, t);
    }
}

// Resource probe (run_vm_probe): for every tile - one instruction each - every warp writes the CTA's tensor-memory base
// + 1 into its two slots, so the host sees that all eight warps took part in every instruction and that the allocation
// they saw never changed.
__device__ __forceinline__ void probe_instruction(const VmProgram& prog, Ctl* ctl, const StageDesc& st, uint32_t tmem, int first, int count) {
    const ProbeParams& p = st.p.probe;
    const int warp = threadIdx.x >> 5;
    for (int t = first; t < first + count; ++t) {
        if (lane_id() == 0) {
            p.out[t * 16 + warp] = static_cast<int>(tmem) + 1;
            p.out[t * 16 + warp + 8] = static_cast<int>(tmem) + 1;
        }
        cta_publish_tile(prog, st, t);
    }
}

}  // namespace pi0
