// Cluster primitives of the single-lattice kernels (cluster.cu,
// cluster_deep.cu): bounded mbarrier waits, remote arrivals and asynchronous
// remote stores, the hardware cluster barrier's halves.
#pragma once

#include <stdint.h>

#define XK_CL_WAIT_NS 1000000000ull   // a CTA gives up after 1 s of waiting (never expected)

__device__ __forceinline__ bool xk_cl_try_wait(uint32_t bar, uint32_t parity)
{
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return done != 0;
}

__device__ __forceinline__ uint64_t xk_globaltimer()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// wait for the phase of `parity` to complete; false after XK_CL_WAIT_NS
__device__ __forceinline__ bool xk_cl_wait(uint32_t bar, uint32_t parity)
{
    if (xk_cl_try_wait(bar, parity)) return true;
    const uint64_t t0 = xk_globaltimer();
    while (!xk_cl_try_wait(bar, parity))
        if (xk_globaltimer() - t0 > XK_CL_WAIT_NS) return false;
    return true;
}

// arrive on the mbarrier at shared::cluster address `bar` (another CTA's),
// ordering this thread's earlier stores before it
__device__ __forceinline__ void xk_cl_arrive_remote(uint32_t bar)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" : : "r"(bar) : "memory");
}

// store v at shared::cluster address `addr` (another CTA's) asynchronously;
// its completion counts 4 bytes on the mbarrier at shared::cluster address
// `bar` of the same CTA
__device__ __forceinline__ void xk_cl_st_async(uint32_t addr, uint32_t v, uint32_t bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];"
                 : : "r"(addr), "r"(v), "r"(bar) : "memory");
}

// this CTA's arrival on its own mbarrier, expecting `bytes` of transactions
__device__ __forceinline__ void xk_cl_arm(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" : : "r"(bar), "r"(bytes) : "memory");
}

// the hardware cluster barrier's two halves (every thread of every CTA
// alternates them)
__device__ __forceinline__ void xk_cl_barrier_arrive()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" : : : "memory");
}

__device__ __forceinline__ void xk_cl_barrier_wait()
{
    asm volatile("barrier.cluster.wait.acquire.aligned;" : : : "memory");
}

__device__ __forceinline__ uint32_t xk_cl_mapa(uint32_t addr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
