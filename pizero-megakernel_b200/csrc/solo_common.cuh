// Bounded waits and the pair-of-CTAs forms of the tcgen05 / TMA wrappers, for the kernels of single operators.
#pragma once
#include "ptx.cuh"
#include "vm_types.h"

namespace pi0 {

// ---------------------------------------------------------------- bounded waits
struct SoloWait {
    VmStatus* status;
    unsigned long long budget_ns;
    int* abort;                  // shared memory: somebody of this CTA has given up
};
// Out of time: recorded for the host, and every other wait of the CTA, and of the operator's other CTAs, ends.  (The first reporter wins.)
static __device__ __noinline__ bool solo_give_up(SoloWait w, uint32_t parity) {
    if (atomicCAS(&w.status->code, 0, 2) == 0) {
        w.status->worker = static_cast<int>(blockIdx.x);
        w.status->stage = 0;
        w.status->band = -1;
        w.status->observed = parity;
        w.status->expected = 0;
        __threadfence();
    }
    atomicExch(&w.status->abort, 1);
    *reinterpret_cast<volatile int*>(w.abort) = 1;
    return false;
}
// Whether a wait of this CTA has run out: its tile is not complete, and nobody may be told that it is.
__device__ __forceinline__ bool solo_gave_up(const int* abort) { return *reinterpret_cast<const volatile int*>(abort) != 0; }
template <bool CLUSTER>
__device__ __forceinline__ bool solo_try(uint64_t* bar, uint32_t parity) {
    if constexpr (!CLUSTER) return mbar_try_wait(bar, parity);
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(1000u) : "memory");
    return ok != 0;
}
// The time of a wait begins behind the kernel in front, which issuing warps do not wait for themselves (a dependency in front of their loops made q|k|v of
// 51 rows 4.17 us, here 4.11), and is looked at from the second round of tries on: a poll of the operator's flag is a trip to L2.
template <bool CLUSTER>
static __device__ __noinline__ bool solo_wait_long(SoloWait w, uint64_t* bar, uint32_t parity) {
    unsigned long long start = 0;
    for (uint32_t spin = 1;; ++spin) {
        if (solo_try<CLUSTER>(bar, parity)) return true;     // each try suspends for at most ~1 us
        if (solo_gave_up(w.abort)) return false;
        if ((spin & 15u) == 0u) {
            if (start == 0) {
                grid_dependency_wait();
                start = global_ns();
            } else if (global_ns() - start > w.budget_ns || ld_relaxed_int(&w.status->abort)) {
                return solo_give_up(w, parity);
            }
        }
    }
}
// One thread.
__device__ __forceinline__ bool solo_wait(const SoloWait& w, uint64_t* bar, uint32_t parity) {
    return mbar_try_wait(bar, parity) || solo_wait_long<false>(w, bar, parity);
}
// One thread, on a barrier that the other CTA of the pair arrives on too.
template <int CG>
__device__ __forceinline__ bool solo_wait_cluster(const SoloWait& w, uint64_t* bar, uint32_t parity) {
    return solo_try<CG == 2>(bar, parity) || solo_wait_long<CG == 2>(w, bar, parity);
}
// A whole warp: one decision for all lanes, each of which has seen the phase complete.
static __device__ __noinline__ bool solo_wait_warp_long(SoloWait w, uint64_t* bar, uint32_t parity) {
    unsigned long long start = 0;
    for (uint32_t spin = 1;; ++spin) {
        if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
        int stop = 0;
        if (lane_id() == 0) {
            if (solo_gave_up(w.abort)) stop = 1;
            else if ((spin & 15u) == 0u) {
                if (start == 0) start = global_ns();
                else if (global_ns() - start > w.budget_ns || ld_relaxed_int(&w.status->abort)) { solo_give_up(w, parity); stop = 1; }
            }
        }
        if (__shfl_sync(0xffffffffu, stop, 0)) return false;
    }
}
__device__ __forceinline__ bool solo_wait_warp(const SoloWait& w, uint64_t* bar, uint32_t parity) {
    return __all_sync(0xffffffffu, mbar_try_wait(bar, parity)) || solo_wait_warp_long(w, bar, parity);
}

// ---------------------------------------------------------------- clusters
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of the same shared-memory location in another CTA of the cluster.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void st_cluster_int(uint32_t addr, int v) {
    asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
// (relaxed: what it tells is that tensor memory has been read, and tcgen05.wait::ld has returned; a release would wait for the draining warp's stores)
__device__ __forceinline__ void mbar_arrive_remote(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cta.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// ---------------------------------------------------------------- TMA into this CTA's memory; in a pair the barrier may be the other's
template <int CG>
__device__ __forceinline__ void tma_load_2d_cg(void* dst, const void* tmap, uint32_t bar, int x, int y) {
    if constexpr (CG == 2)
        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
                     "l"(tmap), "r"(bar), "r"(x), "r"(y) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)), "l"(tmap),
                     "r"(bar), "r"(x), "r"(y) : "memory");
}
template <int CG>
__device__ __forceinline__ void tma_load_3d_cg(void* dst, const void* tmap, uint32_t bar, int x, int y, int z) {
    if constexpr (CG == 2)
        asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
                     "l"(tmap), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)), "l"(tmap),
                     "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
template <int CG>
__device__ __forceinline__ void tma_load_4d_cg(void* dst, const void* tmap, uint32_t bar, int x, int y, int z, int v) {
    if constexpr (CG == 2)
        asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(
                         smem_u32(dst)), "l"(tmap), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(v) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smem_u32(dst)),
                     "l"(tmap), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(v) : "memory");
}

// A box of shared memory to global; and until this thread's stores are complete.
__device__ __forceinline__ void tma_store_2d(const void* tmap, const void* src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(tmap), "r"(smem_u32(src)), "r"(x), "r"(y) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void tma_store_3d(const void* tmap, const void* src, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(tmap), "r"(smem_u32(src)), "r"(x), "r"(y), "r"(z) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_store_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ---------------------------------------------------------------- tcgen05 (a kernel uses one cta_group throughout)
template <int CG>
__device__ __forceinline__ void tmem_alloc_cg(uint32_t* dst_in_smem, uint32_t cols) {
    if constexpr (CG == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_in_smem)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
        tmem_alloc(dst_in_smem, cols);
        tmem_relinquish();
    }
}
template <int CG>
__device__ __forceinline__ void tmem_dealloc_cg(uint32_t taddr, uint32_t cols) {
    if constexpr (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
    else tmem_dealloc(taddr, cols);
}
// Arrive on this barrier (of both CTAs of a pair, `both` being their places in the cluster) once everything issued so far has been done.
template <int CG>
__device__ __forceinline__ void tc_commit_cg(uint64_t* bar, uint16_t both) {
    if constexpr (CG == 2)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                     "h"(both) : "memory");
    else tc_commit(bar);
}
// (in a pair: each CTA's tensor memory from its own shared memory)
template <int CG>
__device__ __forceinline__ void tc_copy_sf_cg(uint32_t taddr, uint64_t sdesc) {
    if constexpr (CG == 2) asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
    else tc_copy_sf(taddr, sdesc);
}
template <int CG>
__device__ __forceinline__ void tc_mma_nvfp4_cg(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
    if constexpr (CG == 2)
        asm volatile(
            "{ .reg .pred p; setp.ne.b32 p, %6, 0;\n"
            "  tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%4], [%5], p; }" ::"r"(d),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate) : "memory");
    else tc_mma_nvfp4(d, adesc, bdesc, idesc, sfa, sfb, accumulate);
}
template <int CG, bool FP8>
__device__ __forceinline__ void tc_mma_dense_cg(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    if constexpr (CG == 2 && FP8)
        asm volatile(
            "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
            "  tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p; }" ::"r"(d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
    else if constexpr (CG == 2)
        asm volatile(
            "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
            "  tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
    else if constexpr (FP8) tc_mma_f8(d, adesc, bdesc, idesc, accumulate);
    else tc_mma_f16(d, adesc, bdesc, idesc, accumulate);
}

}  // namespace pi0
