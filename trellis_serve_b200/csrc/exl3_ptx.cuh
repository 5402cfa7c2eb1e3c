// Thin wrappers over the sm_90+/sm_100 PTX used by the kernels: mbarrier, 1-D bulk async copy (TMA engine,
// no multicast), clusters, counters, named barriers.  Every wait is bounded: it returns false after a fixed time (MBAR_MAX_NS) instead
// of spinning forever, and the caller records the failure in the device error word.
#pragma once
#include <cstdint>

namespace exl3 {
namespace ptx {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_fence_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

// A waiting warp is suspended by the hardware until the phase completes or a time of its own choosing has passed.  (Giving it a
// time hint instead compiles into a polling loop with sleeps.)
__device__ __forceinline__ bool mbar_try_wait_addr(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) { return mbar_try_wait_addr(smem_addr(bar), parity); }

// Bounded waits: how long a failed poll suspends the warp is up to the hardware, so the bound is a time, not a number of polls.
constexpr uint64_t MBAR_MAX_NS = 2000000000ull;

__device__ __forceinline__ uint64_t time_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity)
{
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = time_ns();
    do {
        if (mbar_try_wait(bar, parity)) return true;
    } while (time_ns() - t0 < MBAR_MAX_NS);
    return false;
}

// For a thread that is in no hurry (a copy producer far ahead of its consumers): sleeps between polls so that it does not take
// issue slots from the warps doing the work.
__device__ __forceinline__ bool mbar_wait_relaxed(uint64_t* bar, uint32_t parity, uint32_t sleep_ns = 256)
{
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = time_ns();
    do {
        __nanosleep(sleep_ns);
        if (mbar_try_wait(bar, parity)) return true;
    } while (time_ns() - t0 < MBAR_MAX_NS);
    return false;
}

// ---- thread-block clusters: a barrier of the other CTA of a pair, and the cluster-wide barrier
__device__ __forceinline__ uint32_t cluster_cta_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// All threads of every CTA of the cluster (convergent warps).
__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Arrive on the barrier at the same shared-memory offset in CTA `cta` of the cluster.
__device__ __forceinline__ void mbar_arrive_cluster(uint64_t* bar, uint32_t cta)
{
    asm volatile("{\n .reg .b32 ra;\n mapa.shared::cluster.u32 ra, %0, %1;\n mbarrier.arrive.release.cluster.shared::cluster.b64 _, [ra];\n}" ::"r"(
                     smem_addr(bar)),
                 "r"(cta)
                 : "memory");
}

// Floats at the same shared-memory offset in CTA `cta` of the cluster.
__device__ __forceinline__ float ld_shared_cluster_f32(const float* p, uint32_t cta)
{
    float v;
    asm volatile("{\n .reg .b32 ra;\n mapa.shared::cluster.u32 ra, %1, %2;\n ld.shared::cluster.f32 %0, [ra];\n}" : "=f"(v) : "r"(smem_addr(p)), "r"(cta) : "memory");
    return v;
}
__device__ __forceinline__ float4 ld_shared_cluster_f32x4(const float* p, uint32_t cta)
{
    float4 v;
    asm volatile("{\n .reg .b32 ra;\n mapa.shared::cluster.u32 ra, %4, %5;\n ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [ra];\n}"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(smem_addr(p)), "r"(cta) : "memory");
    return v;
}

// The word at the same shared-memory offset in CTA `cta` of the cluster.
__device__ __forceinline__ int ld_shared_cluster_s32(const int* p, uint32_t cta)
{
    int v;
    asm volatile("{\n .reg .b32 ra;\n mapa.shared::cluster.u32 ra, %1, %2;\n ld.shared::cluster.s32 %0, [ra];\n}" : "=r"(v) : "r"(smem_addr(p)), "r"(cta) : "memory");
    return v;
}

// Bounded wait on a barrier of this CTA that threads of the other CTA arrive on.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity)
{
    const uint64_t t0 = time_ns();
    do {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
    } while (time_ns() - t0 < MBAR_MAX_NS);
    return false;
}

// Global counter update with acquire-release semantics between the CTAs of the device.
__device__ __forceinline__ int atom_add_acq_rel_gpu(int* addr, int v)
{
    int old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(addr), "r"(v) : "memory");
    return old;
}

// Single 64-bit accesses at system scope: the unit of the tagged-word exchange between GPUs (value + call number
// arrive together, so the receiver needs no fence and no separate flag).
__device__ __forceinline__ void st_relaxed_sys_u64(unsigned long long* p, unsigned long long v)
{
    asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed_sys_u64(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Two adjacent tagged words in one 16-byte access (each 8-byte half is what has to arrive whole): a warp then writes
// full 128-byte lines over NVLink instead of half-filled ones.
__device__ __forceinline__ void st_relaxed_sys_v2u64(unsigned long long* p, unsigned long long a, unsigned long long b)
{
    asm volatile("st.relaxed.sys.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void ld_relaxed_sys_v2u64(const unsigned long long* p, unsigned long long& a, unsigned long long& b)
{
    asm volatile("ld.relaxed.sys.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}

// global -> shared bulk copy through the TMA engine; completion is counted in bytes on `bar`.
// Both addresses 16-byte aligned, size a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* smem_dst, const void* gmem_src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(smem_dst)),
                 "l"(gmem_src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

// 1-D bulk copy shared -> global (16-byte aligned on both sides, size a multiple of 16), tracked by the issuing thread's
// bulk groups: commit, then wait until the source may be overwritten (.read) or until the copies have completed.
__device__ __forceinline__ void bulk_s2g(void* gmem_dst, const void* smem_src, uint32_t bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gmem_dst), "r"(smem_addr(smem_src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Programmatic dependent launch: a kernel launched with the programmatic-serialization attribute may start before
// the kernel ahead of it in the stream has finished.  `grid_dependency_wait` blocks until that kernel has completed
// and its writes are visible; `grid_launch_dependents` lets the next kernel in the stream start its own prologue.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void named_bar_sync(int id, int threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ uint32_t lds32(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

__device__ __forceinline__ uint2 lds64(uint32_t addr)
{
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}

__device__ __forceinline__ uint4 lds128(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

}  // namespace ptx
}  // namespace exl3
