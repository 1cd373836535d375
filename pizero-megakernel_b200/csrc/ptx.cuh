// Thin inline-PTX wrappers for sm_100a: mbarrier, TMA (bulk tensor loads), tcgen05
// (TMEM allocation, block-scaled MMA, scale-factor copies, accumulator loads),
// acquire/release counters and the FP4/FP8 converters.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <stdint.h>

namespace pi0 {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
// Pull a 128-byte line of constant data (tables, norm weights) towards this SM ahead of its use.
__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
// A value every lane of the warp holds, in a form the compiler can see is warp-uniform (broadcast from lane 0), so
// arithmetic on it runs on the uniform datapath and tcgen05 operands need no per-instruction register transfers.
__device__ __forceinline__ uint32_t uniform_u32(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ int uniform_i32(int v) { return __shfl_sync(0xffffffffu, v, 0); }
// One lane of a converged warp (always the same one for the full mask).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{ .reg .pred P; elect.sync _|P, 0xffffffff; selp.u32 %0, 1, 0, P; }" : "=r"(p));
    return p != 0;
}

// Programmatic dependent launch: returns when every grid in front of this one in the stream has completed and its writes
// are visible.  (Without the launch attribute it returns at once.)
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Once every CTA has said this (or exited), CTAs of the next grid may take up free SMs and prepare; that grid's own
// grid_dependency_wait still waits for this one's end.
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_count(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
// One try of a phase wait. The thread may be suspended inside the instruction; the explicit hint bounds that
// suspension to about a microsecond (without it the limit is system dependent and can be very long), so a caller
// that polls an abort flag between tries stays responsive. A completing phase wakes the thread immediately.
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(1000u)
        : "memory");
    return ok != 0;
}

// Whether a phase is complete, without waiting.
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}

// ---------------------------------------------------------------- proxies / fences
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_load_2d(void* dst, const void* tmap, uint64_t* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"(tmap), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const void* tmap, uint64_t* bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"(tmap), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}
// Plain (untiled) bulk copy global -> shared; both addresses 16-byte aligned, size a multiple of 16.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void prefetch_tmap(const void* tmap) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}

// ---------------------------------------------------------------- tcgen05 / TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_in_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_in_smem)), "r"(cols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
// Shared-memory matrix descriptor, K-major operand tile with 128-byte swizzle:
// rows are 128 bytes, 8-row groups are 1024 bytes apart (SBO), descriptor version 1.
__device__ __forceinline__ uint64_t umma_desc_k_sw128(uint32_t saddr) {
    return static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// Descriptor of a 32-line x 16-byte scale-factor atom (no swizzle, 8-line groups 128 bytes apart).
__device__ __forceinline__ uint64_t umma_desc_sf(uint32_t saddr) {
    return static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | (8ull << 32) | (1ull << 46);
}
__device__ __forceinline__ void tc_copy_sf(uint32_t taddr, uint64_t sdesc) {
    asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
__device__ __forceinline__ void tc_mma_nvfp4(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t sfa,
                                             uint32_t sfb, uint32_t accumulate) {
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, %6, 0;\n"
        "  tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%4], [%5], p; }" ::"r"(d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
        : "memory");
}
// Dense operands, FP32 accumulator: BF16 x BF16 (K = 16 per instruction) and E4M3 x E4M3 (K = 32 per instruction).
__device__ __forceinline__ void tc_mma_f16(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
        "  tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tc_mma_f8(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
        "  tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p; }" ::"r"(d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp receives lane (row) base+i.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 4 x 4 transpose of 16-byte pieces inside every group of four lanes (its own inverse): lane j's piece k <-> lane k's piece j.
// A drain holds one row per lane; 64 bytes per lane stored row by row touch 32 lines per instruction, and the load / store
// unit takes one line a cycle (128 x 128 BF16 tiles: 1 us of 3.1 per tile).  Transposed, four lanes cover one row's 64
// bytes and an instruction eight rows.
// PIECES: whole 16-byte pieces per step instead of word by word, for the split attention tiles of the lean variants without 192-wide
// tiles (prefix attention of 784 rows 29.4 -> 28.8 us, of 768 rows 17.9 -> 17.8).  In the drains and in the other variants
// word by word is as fast or faster, with fewer registers (three views 8.98 ms, 9.01 with pieces; BF16 16.08 and 16.28).
template <bool PIECES>
__device__ __forceinline__ void quad_transpose(uint4 (&p)[4]) {
    if constexpr (PIECES) {
#pragma unroll
        for (int bit = 1; bit <= 2; bit <<= 1) {
            const bool upper = (lane_id() & bit) != 0;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (i & bit) continue;
                uint4 &lo = p[i], &hi = p[i + bit];
                const uint4 send = upper ? lo : hi;
                const uint4 got = make_uint4(__shfl_xor_sync(0xffffffffu, send.x, bit), __shfl_xor_sync(0xffffffffu, send.y, bit),
                                             __shfl_xor_sync(0xffffffffu, send.z, bit), __shfl_xor_sync(0xffffffffu, send.w, bit));
                if (upper) lo = got;
                else hi = got;
            }
        }
        return;
    }
    const bool odd = (lane_id() & 1) != 0, high = (lane_id() & 2) != 0;
#pragma unroll
    for (int w = 0; w < 4; w++) {
        uint32_t a[4];
#pragma unroll
        for (int i = 0; i < 4; i++) a[i] = w == 0 ? p[i].x : w == 1 ? p[i].y : w == 2 ? p[i].z : p[i].w;
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
            const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? a[i] : a[i + 1], 1);
            if (odd) a[i] = got; else a[i + 1] = got;
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const uint32_t got = __shfl_xor_sync(0xffffffffu, high ? a[i] : a[i + 2], 2);
            if (high) a[i] = got; else a[i + 2] = got;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) (w == 0 ? p[i].x : w == 1 ? p[i].y : w == 2 ? p[i].z : p[i].w) = a[i];
    }
}
// Whole warp: lane r holds 64 bytes of row r (r < rows), `own` is where they belong, rows are `ld` bytes apart.
template <bool PIECES = false>
__device__ __forceinline__ void store_rows64(uint8_t* own, int ld, int rows, uint4 (&p)[4]) {
    quad_transpose<PIECES>(p);
    const int lane = lane_id(), mine = lane & 3;
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (lane - mine + k < rows) *reinterpret_cast<uint4*>(own + static_cast<ptrdiff_t>(k - mine) * ld + mine * 16) = p[k];
}

// ---------------------------------------------------------------- counters
__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int ld_relaxed_int(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release_add(unsigned int* p, unsigned int v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void named_barrier(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// ---------------------------------------------------------------- number formats
// Pairs of FP32 operations in one instruction, each lane rounded as its scalar form.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(d)
        : "l"(*reinterpret_cast<const uint64_t*>(&a)), "l"(*reinterpret_cast<const uint64_t*>(&b)), "l"(*reinterpret_cast<const uint64_t*>(&c)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<const uint64_t*>(&a)), "l"(*reinterpret_cast<const uint64_t*>(&b)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<const uint64_t*>(&a)), "l"(*reinterpret_cast<const uint64_t*>(&b)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
    float d;
    asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// 2^x.  The results of exp2f bit for bit where they are normal numbers (compared for every FP32 x from -150 to 0); smaller ones become
// zero.  Its callers have subtracted the maximum, so the largest weight is 1 and the loss of another is below 2^-126.
__device__ __forceinline__ float exp2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Eight FP32 -> four bytes of E2M1 codes (RNE, saturating), the first value in the lowest nibble.
__device__ __forceinline__ uint32_t cvt_e2m1x8(float2 a, float2 b, float2 c, float2 d) {
    uint32_t w;
    asm("{ .reg .b8 p, q, r, s; cvt.rn.satfinite.e2m1x2.f32 p, %2, %1; cvt.rn.satfinite.e2m1x2.f32 q, %4, %3;\n"
        "  cvt.rn.satfinite.e2m1x2.f32 r, %6, %5; cvt.rn.satfinite.e2m1x2.f32 s, %8, %7; mov.b32 %0, {p, q, r, s}; }"
        : "=r"(w) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y), "f"(d.x), "f"(d.y));
    return w;
}
__device__ __forceinline__ uint32_t encode_ue4m3(float x) {
    return static_cast<uint32_t>(__nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3));
}
__device__ __forceinline__ float decode_ue4m3(uint32_t code) {
    __half_raw h = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(code), __NV_E4M3);
    return __half2float(__half(h));
}
// Block scale code for a 16-element block with magnitude maximum `amax`.
// policy 0: nearest-even code of amax*(1/6); policy 1: smallest code not below it.
__device__ __forceinline__ uint32_t block_scale_code(float amax, int policy) {
    float desired = amax * (1.f / 6.f);
    uint32_t code = encode_ue4m3(desired);
    if (policy == 1 && decode_ue4m3(code) < desired && code < 126u) code += 1u;
    return code;
}
// Quantise 16 values (already divided by the tensor scale) -> 8 bytes + scale code.  Few-row operators run this once per
// thread as straight-line code, so its length is their time: packed multiplies, three-input maxima and whole-word
// packing of the codes make it about half as long as the scalar form.
__device__ __forceinline__ uint2 quantize_block16(const float2 (&v)[8], int policy, uint32_t& code_out) {
    const float a = max3_abs(max3_abs(v[0].x, v[0].y, v[1].x), max3_abs(v[1].y, v[2].x, v[2].y), max3_abs(v[3].x, v[3].y, v[4].x));
    // (the zero costs nothing and keeps the maximum a number: the three-input maxima pass over NaNs, but a block of nothing else
    // would hand its NaN on to the scale)
    const float amax = max3_abs(max3_abs(a, v[4].y, v[5].x), max3_abs(v[5].y, v[6].x, v[6].y), max3_abs(v[7].x, v[7].y, 0.f));
    const uint32_t code = block_scale_code(amax, policy);
    const float decoded = decode_ue4m3(code);
    const float recip = decoded > 0.f ? __frcp_rn(decoded) : 0.f;
    const float2 r2 = make_float2(recip, recip);
    float2 s[8];
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = mul2(v[i], r2);
    code_out = code;
    const uint32_t keep = decoded > 0.f ? 0xffffffffu : 0u;            // zero codes (no negative zeros) under a zero scale
    return make_uint2(cvt_e2m1x8(s[0], s[1], s[2], s[3]) & keep, cvt_e2m1x8(s[4], s[5], s[6], s[7]) & keep);
}
__device__ __forceinline__ uint2 quantize_block16(const float (&v)[16], int policy, uint32_t& code_out) {
    float2 pairs[8];
#pragma unroll
    for (int i = 0; i < 8; i++) pairs[i] = make_float2(v[2 * i], v[2 * i + 1]);
    return quantize_block16(pairs, policy, code_out);
}
// Offset of scale (row, block) in the 128x4 atom layout with `blocks` blocks per row.
__device__ __forceinline__ size_t scale_offset(int row, int block, int blocks) {
    return (static_cast<size_t>(row >> 7) * ((blocks + 3) >> 2) + (block >> 2)) * 512 + (row & 31) * 16 +
           ((row & 127) >> 5) * 4 + (block & 3);
}

__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float gelu_tanh(float x) {
    // 0.5 x (1 + tanh(sqrt(2/pi) (x + 0.044715 x^3)))
    float inner = 0.7978845608028654f * (x + 0.044715f * x * x * x);
    return 0.5f * x * (1.f + tanhf(inner));
}

}  // namespace pi0
