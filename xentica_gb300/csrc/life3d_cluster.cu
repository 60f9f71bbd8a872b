// A 3-D von Neumann Life-like lattice, bit-packed along x, in the shared memory
// of a thread-block cluster for all generations of a launch.
//
// The planes are cut into slabs, one a CTA.  A CTA keeps its slab twice
// (ping-pong) with the plane below and above it: a generation reads one copy,
// writes the other, stores the slab's first and last plane into the
// neighbouring CTAs' halos as well, and ends with the hardware cluster
// barrier.  A thread owns a column (one word of a row) over a run of planes
// and walks up it with the words below, at and above in registers: a word
// costs one new load along z and four beside it.
//
// Served lattices: many requests run at once, and a generation of one is a
// launch of its own elsewhere (xk_k_life3d_vn); 9 such requests made 8500 of
// the 15 700 launches of 32 mixed ones.  Here a request takes a few SMs and one
// launch for many generations: the 32 took 26.2 ms before and 23.6 with it.
// A lattice alone: bound by the cluster barrier, 1.4 to 1.5 us a generation up
// to 32 768 words (64^3 1.51, 160 x 50 x 40 1.38; one launch a generation, whose
// launches overlap, 1.63 and 1.89; 4.5 with the kernel of any neighbourhood);
// beyond, by the words its 16 SMs work through: 128^3 2.2 against 1.7.
#include <string.h>

#include <algorithm>

#include "cluster.cuh"
#include "life_word.cuh"

#define XK_L3_THREADS 1024

__device__ __forceinline__ void xk_l3_store_remote(uint32_t addr, uint32_t v)
{
    asm volatile("st.shared::cluster.u32 [%0], %1;" : : "r"(addr), "r"(v) : "memory");
}

template <bool TORUS>
__global__ void __launch_bounds__(XK_L3_THREADS, 1)
xk_k_life3d_cluster(uint32_t *__restrict__ cells, Life3Geo g, const __grid_constant__ LifeTable t, int C,
                    int most, int gens)
{
    extern __shared__ uint32_t sm[];
    const int rank = blockIdx.x, tid = threadIdx.x;     // the grid is one cluster
    const int P = g.H * g.wpr;                          // words of a plane
    const int z0 = (int)((int64_t)rank * g.D / C), z1 = (int)((int64_t)(rank + 1) * g.D / C), n = z1 - z0;
    const int buf = (most + 2) * P;                     // words of a copy: halo, up to `most` planes, halo
    const int prev = rank > 0 ? rank - 1 : C - 1, next = rank + 1 < C ? rank + 1 : 0;
    const int nprev = (int)((int64_t)(prev + 1) * g.D / C) - (int)((int64_t)prev * g.D / C);
    const uint32_t own = (uint32_t)__cvta_generic_to_shared(sm);
    const uint32_t to_prev = xk_cl_mapa(own, prev) + 4u * (uint32_t)((nprev + 1) * P);
    const uint32_t to_next = xk_cl_mapa(own, next);
    for (int w = tid; w < n * P; w += XK_L3_THREADS) sm[P + w] = cells[(int64_t)z0 * P + w];
    for (int w = tid; w < P; w += XK_L3_THREADS) {
        uint32_t below = cells[(int64_t)(z0 > 0 ? z0 - 1 : g.D - 1) * P + w];
        uint32_t above = cells[(int64_t)(z1 < g.D ? z1 : 0) * P + w];
        if (!TORUS) {
            // a border's planes are in both copies: nobody sends them
            if (z0 == 0) sm[buf + w] = below = g.bfill;
            if (z1 == g.D) sm[buf + (n + 1) * P + w] = above = g.bfill;
        }
        sm[w] = below;
        sm[(n + 1) * P + w] = above;
    }
    const bool send_prev = TORUS || rank > 0, send_next = TORUS || rank + 1 < C;
    const uint32_t edge = TORUS ? 0u : g.bfill & 1u;
    // a plane of up to half the threads' columns is walked in several runs
    const int runs = max(1, min(n, XK_L3_THREADS / P));
    const int run = P < XK_L3_THREADS ? tid / P : 0;
    const int za = 1 + run * n / runs, zb = 1 + (run + 1) * n / runs;
    const int c0 = tid - run * P, last = g.wpr - 1;
    xk_cl_barrier_arrive();
    xk_cl_barrier_wait();
    for (int gen = 0; gen < gens; ++gen) {
        const int from = (gen & 1) * buf, into = buf - from;
        if (run < runs)
            for (int col = c0; col < P; col += XK_L3_THREADS) {
                const int y = (int)xk_divu((uint32_t)col, (uint32_t)g.wpr, g.div_wpr), j = col - y * g.wpr;
                const int l = j > 0 ? -1 : last, r = j < last ? 1 : -last;
                const int u = y > 0 ? -g.wpr : (g.H - 1) * g.wpr, d = y + 1 < g.H ? g.wpr : -(g.H - 1) * g.wpr;
                const int lshift = j > 0 ? 31 : g.rlast - 1, top = j == last ? g.rlast - 1 : 31;
                const uint32_t mask = j == last ? g.lastmask : 0xFFFFFFFFu;
                const uint32_t *s = sm + from + za * P + col;
                uint32_t *o = sm + into + za * P + col;
                uint32_t below = s[-P], at = s[0];
#pragma unroll 2
                for (int z = za; z < zb; ++z) {
                    const uint32_t above = s[P];
                    uint32_t U = s[u], Dn = s[d];
                    if (!TORUS) {
                        U = y > 0 ? U : g.bfill;
                        Dn = y + 1 < g.H ? Dn : g.bfill;
                    }
                    const RowVec v = xk_row_vec(at, s[l], s[r], lshift, top, edge, edge, !TORUS && j == 0,
                                                !TORUS && j == last);
                    const uint32_t s1 = xk_lop3_xor3(v.L, v.R, U), c1 = xk_maj(v.L, v.R, U);
                    const uint32_t s2 = xk_lop3_xor3(Dn, below, above), c2 = xk_maj(Dn, below, above);
                    const uint32_t out = xk_life_vn6(t, s1 ^ s2, c1, c2, s1 & s2, at) & mask;
                    *o = out;
                    if (z == 1 && send_prev) xk_l3_store_remote(to_prev + 4u * (uint32_t)(into + col), out);
                    if (z == n && send_next) xk_l3_store_remote(to_next + 4u * (uint32_t)(into + col), out);
                    below = at;
                    at = above;
                    s += P;
                    o += P;
                }
            }
        xk_cl_barrier_arrive();
        xk_cl_barrier_wait();
    }
    const int from = (gens & 1) * buf;
    for (int w = tid; w < n * P; w += XK_L3_THREADS) cells[(int64_t)z0 * P + w] = sm[from + P + w];
}

static void l3_cfg(cudaLaunchConfig_t &cfg, cudaLaunchAttribute &attr, const Life3ClPlan &p, cudaStream_t s)
{
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(p.C);
    cfg.blockDim = dim3(XK_L3_THREADS);
    cfg.dynamicSmemBytes = (size_t)p.smem;
    cfg.stream = s;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = p.C;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
}

typedef void (*L3Kernel)(uint32_t *, Life3Geo, LifeTable, int, int, int);

static L3Kernel l3_kernel(const Life3Geo &g) { return g.torus ? xk_k_life3d_cluster<true> : xk_k_life3d_cluster<false>; }

static cudaError_t l3_attrs(const Life3Geo &g, int smem)
{
    const void *k = (const void *)l3_kernel(g);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e != cudaSuccess || smem <= 48 * 1024 ? e : xk_smem_attr_at_least(k, smem);
}

int xk_life3d_cluster_plan(const Life3Geo &g, bool alone, Life3ClPlan *out)
{
    const int64_t P = (int64_t)g.H * g.wpr, words = P * g.D;
    if (words > (int64_t)16 * xk_max_smem_optin()) return 0;
    // CTAs of about 2048 words (a microsecond a generation, half of it the
    // barrier), at most 8 of them beside other work, more only where they
    // hold the lattice
    const int enough = alone ? 16 : 8;
    if (alone && words > 2048 * 16) return 0;       // one launch a generation is faster
    for (int C = 1; C <= 16; C *= 2) {
        if (C > g.D) return 0;
        Life3ClPlan p;
        p.C = C;
        p.most = (g.D + C - 1) / C;
        const int64_t smem = 8 * (int64_t)(p.most + 2) * P;
        if (smem > xk_max_smem_optin() || (C < enough && 2 * C <= g.D && words > 2048 * (int64_t)C)) continue;
        p.smem = (int)smem;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr;
        l3_cfg(cfg, attr, p, 0);
        int active = 0;
        if (l3_attrs(g, p.smem) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&active, (const void *)l3_kernel(g), &cfg) != cudaSuccess ||
            active < 1) {
            cudaGetLastError();
            return 0;
        }
        *out = p;
        return 1;
    }
    return 0;
}

cudaError_t xk_life_step3d_cluster(uint32_t *cells, const Life3Geo &g, const LifeTable &t, int generations,
                                   const Life3ClPlan &p, cudaStream_t s)
{
    cudaError_t e = l3_attrs(g, p.smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    l3_cfg(cfg, attr, p, s);
    return cudaLaunchKernelEx(&cfg, l3_kernel(g), cells, g, t, p.C, p.most, generations);
}
