/* cluster_common.cuh — thread-block-cluster pieces of the cluster solver (internal):
 * distributed-shared-memory addresses, stores that signal a remote mbarrier, bounded
 * mbarrier waits, and the cluster-wide barrier. */
#ifndef GSLAM_CLUSTER_COMMON_CUH
#define GSLAM_CLUSTER_COMMON_CUH

#include <stdint.h>

__device__ __forceinline__ unsigned cl_smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

/* the address of this CTA's shared location `a` in CTA `rank` of the cluster */
__device__ __forceinline__ unsigned cl_mapa(unsigned a, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}

__device__ __forceinline__ unsigned cl_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

/* every thread of the cluster: what was written before it is visible after it */
__device__ __forceinline__ void cl_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

/* 8 or 16 bytes to a (remote) shared location; its mbarrier counts the bytes when they
 * have arrived, so a thread that waited for them there reads them */
__device__ __forceinline__ void cl_st_async(unsigned dst, double a, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
                 "l"(__double_as_longlong(a)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cl_st_async2(unsigned dst, double a, double b, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "l"(__double_as_longlong(a)), "l"(__double_as_longlong(b)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cl_st_async4(unsigned dst, float a, float b, float c, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                     dst),
                 "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(__float_as_uint(c)), "r"(0u), "r"(bar)
                 : "memory");
}

/* waits for the phase with this parity, with acquire at cluster scope; false after
 * `limit` clock cycles */
__device__ __forceinline__ bool cl_wait(unsigned bar, unsigned parity, long long limit) {
    const long long t0 = clock64();
    while (true) {
        unsigned ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if (clock64() - t0 > limit) return false;
    }
}

#endif
