// ptx.cuh -- inline PTX for shared-memory barriers, cluster shared memory and
// bulk copies (sm_90+ instructions, used here on sm_100a).
#pragma once
#include <cstdint>

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// address of the same shared-memory location in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init_cluster() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// local arrive (release, CTA scope)
__device__ __forceinline__ void mbar_arrive_local(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait_cta(uint32_t addr, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// 1D bulk copy global -> shared, completion counted on an mbarrier (no multicast)
__device__ __forceinline__ void bulk_g2s(void *dst_smem, const void *src_gmem, uint32_t bytes, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst_smem)),
        "l"(src_gmem), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// One element (8 or 16 bytes) copied global -> shared asynchronously by this
// thread; zero where !valid (the source is then not read)
template <int B> __device__ __forceinline__ void cp_async_el(void *dst_smem, const void *src, bool valid);
template <> __device__ __forceinline__ void cp_async_el<16>(void *dst_smem, const void *src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst_smem)), "l"(src),
                 "r"(valid ? 16 : 0)
                 : "memory");
}
template <> __device__ __forceinline__ void cp_async_el<8>(void *dst_smem, const void *src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst_smem)), "l"(src),
                 "r"(valid ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void st_cluster_v2f32(uint32_t addr, float x, float y) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void st_cluster_v2f64(uint32_t addr, double x, double y) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(x), "d"(y) : "memory");
}
__device__ __forceinline__ void st_cluster_u32(uint32_t addr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_cluster_c(uint32_t addr, float2 v) { st_cluster_v2f32(addr, v.x, v.y); }
__device__ __forceinline__ void st_cluster_c(uint32_t addr, double2 v) { st_cluster_v2f64(addr, v.x, v.y); }

// bounded wait: gives up after `limit` polls and reports false
__device__ __forceinline__ bool mbar_wait_bounded_cta(uint32_t addr, uint32_t parity, uint32_t limit) {
    for (uint32_t it = 0; it < limit; ++it)
        if (mbar_try_wait_cta(addr, parity)) return true;
    return false;
}

// Barrier operations of a whole converged warp, by one predicated lane: a poll
// or arrive executed by all 32 lanes is done lane by lane (137 cycles for a
// poll of a completed phase on a B200, and ~190 for one lane's under a branch
// with the reconvergence after it; 22 this way).  The outcome of a poll is the
// warp's, and the __syncwarp orders the other lanes' accesses with lane 0's.
__device__ __forceinline__ bool mbar_poll_warp_cta(uint32_t addr, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.eq.u32 q, %3, 0;\n\t"
        "setp.ne.u32 p, %3, %3;\n\t"
        "@q mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(addr), "r"(parity), "r"((uint32_t)(threadIdx.x & 31))
        : "memory");
    return __any_sync(0xffffffffu, ok != 0);
}
__device__ __forceinline__ bool mbar_poll_warp_cluster(uint32_t addr, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.eq.u32 q, %3, 0;\n\t"
        "setp.ne.u32 p, %3, %3;\n\t"
        "@q mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(addr), "r"(parity), "r"((uint32_t)(threadIdx.x & 31))
        : "memory");
    return __any_sync(0xffffffffu, ok != 0);
}
__device__ __forceinline__ bool mbar_wait_warp_cta(uint32_t addr, uint32_t parity, uint32_t limit) {
    for (uint32_t it = 0; it < limit; ++it)
        if (mbar_poll_warp_cta(addr, parity)) {
            __syncwarp();
            return true;
        }
    return false;
}
__device__ __forceinline__ bool mbar_wait_warp_cluster(uint32_t addr, uint32_t parity, uint32_t limit) {
    for (uint32_t it = 0; it < limit; ++it)
        if (mbar_poll_warp_cluster(addr, parity)) {
            __syncwarp();
            return true;
        }
    return false;
}
// one arrive for the warp, after every lane's earlier accesses
__device__ __forceinline__ void mbar_arrive_warp(uint64_t *bar) {
    __syncwarp();
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.eq.u32 q, %1, 0;\n\t"
        "@q mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(smem_u32(bar)),
        "r"((uint32_t)(threadIdx.x & 31))
        : "memory");
}
__device__ __forceinline__ void mbar_arrive_warp_cluster(uint32_t cluster_addr) {
    __syncwarp();
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.eq.u32 q, %1, 0;\n\t"
        "@q mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n\t}" ::"r"(cluster_addr),
        "r"((uint32_t)(threadIdx.x & 31))
        : "memory");
}
// 16 bytes to shared memory where p, as a predicated store: a branch around a
// few stores costs the warp its reconvergence
__device__ __forceinline__ void st_shared_v4_if(bool p, uint32_t addr, float4 v) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t"
        "@q st.shared.v4.f32 [%1], {%2, %3, %4, %5};\n\t}" ::"r"((uint32_t)p),
        "r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
        : "memory");
}
__device__ __forceinline__ void st_shared_u32_if(bool p, uint32_t addr, uint32_t v) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q st.shared.u32 [%1], %2;\n\t}" ::"r"((uint32_t)p),
                 "r"(addr), "r"(v)
                 : "memory");
}
__device__ __forceinline__ void st_global_f2_if(bool p, float2 *addr, float2 v) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q st.global.v2.f32 [%1], {%2, %3};\n\t}" ::"r"((uint32_t)p),
                 "l"(addr), "f"(v.x), "f"(v.y)
                 : "memory");
}

// this thread's warp in its (1-D) block, in a form the compiler knows to be warp-uniform
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// A position in a ring of `size` slots: the slot, and the parity of the
// current pass over the ring (the phase an mbarrier of the slot completes
// on this use).  Advanced by one per use, without divisions.
struct RingPos {
    int slot = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void next(int size) {
        if (++slot == size) {
            slot = 0;
            phase ^= 1u;
        }
    }
};
