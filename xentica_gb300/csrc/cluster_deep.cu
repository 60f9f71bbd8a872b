// One Life-like lattice (W <= 1024) on a thread-block cluster, rows exchanged
// every XK_DEEP generations.
//
// The rows of a bit-packed lattice are cut into C slabs of R rows, one per CTA
// of a cluster of C (up to 16) CTAs, as in cluster.cu, but a CTA also keeps
// K = XK_DEEP rows of the slabs above and below its own: K generations later
// its own rows are still exact (a cell depends on cells within one row per
// generation), and only then are K fresh rows sent each way.  cluster.cu sends
// a row each way every generation, whose latency through distributed shared
// memory (about 500 cycles) was two thirds of a generation.
//
// A lane group of P = next_pow2(wpr) lanes holds a band of B rows in
// registers, lane j column word j, for the whole launch.  A generation reads
// only the bands' edge rows from shared memory (double-buffered by generation,
// one __syncthreads each), the words beside a lane's by shuffles.  Rows
// farther out than the exact ones compute on whatever is there.
//
// Exchange: rows K .. 2 K - 1 of a CTA's window (the first of its slab) go to
// the CTA above as the rows below its slab, rows R .. R + K - 1 (its last) to
// the CTA below, as asynchronous remote stores that count bytes on the
// receiver's mbarrier of the exchange's parity; thread 0 arms that mbarrier
// once per exchange (one arrival expecting the 8 K wpr bytes; a store may land
// before it: the phase still needs the arrival).  The receiver's lanes that
// hold halo rows take them from the landing area, double-buffered by the same
// parity.  A CTA sends exchange e + 2 only after it has received its
// neighbours' e + 1, which they sent after reading their landing areas of e.
// Waits are bounded (1 s): a CTA that gives up sets *gave_up, leaves the loop
// with all its threads and waits as long once more for rows that are still on
// their way; the last cluster barrier keeps every CTA's shared memory alive
// until all are done.
//
// Microseconds a generation, Conway's rule compiled in, 16 CTAs: 512 x 512 0.237
// (cluster.cu 0.362, temporal blocking 0.389), 256 x 256 0.131 (0.329); 1000 x
// 700 0.526 (temporal blocking 0.402, which the tuner keeps there).  Bound by the
// shuffles and shared-memory accesses of a generation.  K = 4: 0.268 at 512 x
// 512, K = 16: 0.277.
#include <string.h>

#include "cluster.cuh"
#include "life_word.cuh"
#include "xk_internal.cuh"

#define XK_DEEP 8

// shared words: bands' edge rows [2][bands][2][P], landing areas
// [2][above, below][K][wpr], then (8-byte aligned) the two mbarriers
static inline int64_t deep_words(int wpr, int P, int bands)
{
    const int64_t w = 4LL * bands * P + 4LL * XK_DEEP * wpr;
    return ((w + 1) & ~1LL) + 4;
}

template <bool TORUS, bool FULLW, int B, int RF>
__global__ void __launch_bounds__(1024)
xk_k_life_deep(uint32_t *__restrict__ bits, LifeGeo g, LifeTable9 t9, int generations, int R, int bands,
               unsigned int *__restrict__ gave_up)
{
    constexpr int K = XK_DEEP;
    const auto &t = RuleForm<RF>::make(t9);
    extern __shared__ uint32_t sm[];
    const int C = (int)gridDim.x, c = (int)blockIdx.x;        // one cluster: rank = block
    const int wpr = g.wpr, H = g.H;
    const int r0 = c * R, Rc = min(H, r0 + R) - r0;          // rows of this CTA (>= K)
    const int cu = c > 0 ? c - 1 : C - 1, cd = c + 1 < C ? c + 1 : 0;
    int P = 1;
    while (P < wpr) P <<= 1;
    const int gpw = 32 / P;
    uint32_t *edge = sm;                                     // [parity][band][first, last][P]
    uint32_t *land = sm + 4 * bands * P;                     // [parity][above, below][K][wpr]
    uint64_t *mbar = (uint64_t *)(sm + ((4LL * bands * P + 4LL * K * wpr + 1) & ~1LL));
    const uint32_t mbar0 = (uint32_t)__cvta_generic_to_shared(mbar);
    if (threadIdx.x == 0) {
        for (int q = 0; q < 2; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" : : "r"(mbar0 + 8u * q) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" : : : "memory");
    }
    const uint32_t land0 = (uint32_t)__cvta_generic_to_shared(land);
    const uint32_t mb_up = xk_cl_mapa(mbar0, (uint32_t)cu), mb_dn = xk_cl_mapa(mbar0, (uint32_t)cd);
    const uint32_t la_up = xk_cl_mapa(land0, (uint32_t)cu), la_dn = xk_cl_mapa(land0, (uint32_t)cd);

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = lane / P, j = lane - q * P;
    const int band = warp * gpw + q;
    // idle lanes (past the row's words, past the bands) compute on a copy of
    // a neighbouring word, so the shuffles always see the whole warp
    const int bc = min(band, bands - 1), jc = min(j, wpr - 1);
    const bool active = band < bands && j < wpr;
    const int last = wpr - 1;
    const int src_l = q * P + (jc > 0 ? jc - 1 : last), src_r = q * P + (jc < last ? jc + 1 : 0);
    const int lshift = jc > 0 ? 31 : g.rlast - 1, lpre = 31 - lshift;
    const int top = jc == last ? g.rlast - 1 : 31;
    const uint32_t topbit = 1u << top;
    const uint32_t outmask = jc == last ? g.lastmask : 0xFFFFFFFFu;
    const uint32_t bedge = g.bfill & 1u;
    const int use_le = !TORUS && jc == 0, use_re = !TORUS && jc == last;
    const int w0 = bc * B;                                   // the band's first window row
    const int y0 = r0 - K + w0;                              // its lattice row

    // the window from global memory: slab and halo rows
    uint32_t w[B];
    {
        int y = y0;
        if (TORUS) {
            y %= H;
            if (y < 0) y += H;
        }
#pragma unroll
        for (int i = 0; i < B; ++i) {
            const bool off = !TORUS && (y < 0 || y >= H);
            w[i] = off ? g.bfill : bits[(int64_t)(off ? 0 : y) * wpr + jc];
            ++y;
            if (TORUS && y == H) y = 0;
        }
    }
    // every CTA running, its mbarriers set, its window read (the slabs are
    // written back only after the last barrier)
    xk_cl_barrier_arrive();
    xk_cl_barrier_wait();

    auto sums = [&](uint32_t v, uint32_t &s, uint32_t &cy) {
        const uint32_t l = __shfl_sync(0xFFFFFFFFu, v, src_l), r = __shfl_sync(0xFFFFFFFFu, v, src_r);
        if (FULLW) {
            const uint32_t L = __funnelshift_l(l, v, 1), Rr = __funnelshift_r(v, r, 1);
            s = xk_lop3_xor3(L, v, Rr);
            cy = xk_maj(L, v, Rr);
            return;
        }
        const RowVec n = TORUS ? xk_torus_vec(v, l, r, lpre, top, topbit)
                               : xk_row_vec(v, l, r, lshift, top, bedge, bedge, use_le, use_re);
        s = xk_lop3_xor3(n.L, n.C, n.R);
        cy = xk_maj(n.L, n.C, n.R);
    };
    auto off_row = [&](int i) { return !TORUS && (y0 + i < 0 || y0 + i >= H); };
    const int stride = bands * 2 * P;
    uint32_t *mine = edge + bc * 2 * P + jc;
    const uint32_t *above = edge + (bc > 0 ? (bc - 1) * 2 + 1 : 0) * P + jc;
    const uint32_t *below = edge + (bc + 1 < bands ? (bc + 1) * 2 : bc * 2 + 1) * P + jc;
    auto generation = [&](int par) {
        if (active) {
            mine[par * stride] = w[0];
            mine[par * stride + P] = w[B - 1];
        }
        __syncthreads();
        uint32_t su, cu_, sm_, cm_, sd, cd_;
        sums(above[par * stride], su, cu_);
        const uint32_t dn = below[par * stride];
        if (off_row(-1)) su = cu_ = g.bfill;
        sums(w[0], sm_, cm_);
        if (off_row(0)) sm_ = cm_ = g.bfill;
#pragma unroll
        for (int i = 0; i < B; ++i) {
            const uint32_t v = w[i];
            sums(i + 1 < B ? w[i + 1 < B ? i + 1 : i] : dn, sd, cd_);
            if (off_row(i + 1)) sd = cd_ = g.bfill;
            uint32_t out = xk_life_word9(su, cu_, sm_, cm_, sd, cd_, v, t);
            if (!FULLW) out &= outmask;
            w[i] = off_row(i) ? g.bfill : out;
            su = sm_;
            cu_ = cm_;
            sm_ = sd;
            cm_ = cd_;
        }
    };

    int left = generations, e = 0;
    for (;; ++e) {
        const int n = min(left, K);
        for (int k = 0; k < n; k += 2) {
            generation(0);
            if (k + 1 < n) generation(1);
        }
        left -= n;
        if (left == 0) break;
        // exchange e
        const uint32_t par = (uint32_t)e & 1u, bar = mbar0 + 8u * par;
        if (threadIdx.x == 0) xk_cl_arm(bar, 8u * K * (uint32_t)wpr);
        if (active) {
#pragma unroll
            for (int i = 0; i < B; ++i) {
                const int r = w0 + i;
                if (r >= K && r < 2 * K)
                    xk_cl_st_async(la_up + 4u * (uint32_t)(((int)par * 2 + 1) * K * wpr + (r - K) * wpr + j), w[i],
                                   mb_up + 8u * par);
                if (r >= Rc && r < Rc + K)
                    xk_cl_st_async(la_dn + 4u * (uint32_t)((int)par * 2 * K * wpr + (r - Rc) * wpr + j), w[i],
                                   mb_dn + 8u * par);
            }
        }
        const bool failed = !xk_cl_wait(bar, (uint32_t)(e >> 1) & 1u);
        if (failed) atomicOr(gave_up, 1u);
        if (__syncthreads_or(failed)) break;
        const uint32_t *from = land + (int)par * 2 * K * wpr;
#pragma unroll
        for (int i = 0; i < B; ++i) {
            const int r = w0 + i;
            if (off_row(i)) continue;
            if (r < K) w[i] = from[r * wpr + jc];
            else if (r >= Rc + K && r < Rc + 2 * K) w[i] = from[K * wpr + (r - Rc - K) * wpr + jc];
        }
        // an even number of generations lies between exchanges, so the edge
        // rows' parities carry on
    }
    // gave up: rows that are still on their way land while the CTA is there
    if (left != 0) xk_cl_wait(mbar0 + 8u * ((uint32_t)e & 1u), (uint32_t)(e >> 1) & 1u);
    xk_cl_barrier_arrive();
    xk_cl_barrier_wait();
    if (!active) return;
#pragma unroll
    for (int i = 0; i < B; ++i) {
        const int r = w0 + i;
        if (r >= K && r < K + Rc) bits[(int64_t)(r0 + r - K) * wpr + j] = w[i];
    }
}

typedef void (*DeepKernel)(uint32_t *, LifeGeo, LifeTable9, int, int, int, unsigned int *);

template <bool TORUS, bool FULLW, int RF>
static DeepKernel deep_kernel_b(int B)
{
    switch (B) {
    case 2: return xk_k_life_deep<TORUS, FULLW, 2, RF>;
    case 3: return xk_k_life_deep<TORUS, FULLW, 3, RF>;
    case 4: return xk_k_life_deep<TORUS, FULLW, 4, RF>;
    case 6: return xk_k_life_deep<TORUS, FULLW, 6, RF>;
    default: return nullptr;
    }
}

template <int RF>
static DeepKernel deep_kernel_rf(const LifeGeo &g, int B)
{
    if (!g.torus) return deep_kernel_b<false, false, RF>(B);
    return g.rlast == 32 ? deep_kernel_b<true, true, RF>(B) : deep_kernel_b<true, false, RF>(B);
}

static DeepKernel deep_kernel(const LifeGeo &g, int B, int rf)
{
    return rf == XK_RULE_CONWAY ? deep_kernel_rf<XK_RULE_CONWAY>(g, B) : deep_kernel_rf<XK_RULE_TABLE>(g, B);
}

static void deep_cfg(cudaLaunchConfig_t &cfg, cudaLaunchAttribute &attr, const DeepPlan &p, cudaStream_t s)
{
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(p.C);
    cfg.blockDim = dim3(p.threads);
    cfg.dynamicSmemBytes = (size_t)p.smem;
    cfg.stream = s;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = p.C;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
}

static cudaError_t deep_attrs(DeepKernel k, int smem)
{
    cudaError_t e = cudaFuncSetAttribute((const void *)k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e != cudaSuccess || smem <= 48 * 1024 ? e : xk_smem_attr_at_least((const void *)k, smem);
}

int xk_life_deep_config(const LifeGeo &g, int C, int B, DeepPlan *out)
{
    if (g.wpr > 32 || C < 2 || C > 16 || !deep_kernel(g, B, XK_RULE_TABLE)) return 0;
    DeepPlan p;
    p.B = B;
    p.R = (g.H + C - 1) / C;
    p.C = (g.H + p.R - 1) / p.R;                             // no empty CTA
    // every slab has the rows its neighbours' halos take
    if (p.C < 2 || g.H - (p.C - 1) * p.R < XK_DEEP) return 0;
    int P = 1;
    while (P < g.wpr) P <<= 1;
    p.bands = (p.R + 2 * XK_DEEP + B - 1) / B;
    const int gpw = 32 / P;
    p.threads = (p.bands + gpw - 1) / gpw * 32;
    if (p.threads > 1024) return 0;
    p.smem = (int)(4 * deep_words(g.wpr, P, p.bands));
    if (p.smem > xk_max_smem_optin()) return 0;
    int active = 0;
    for (int rf = XK_RULE_TABLE; rf <= XK_RULE_CONWAY; ++rf) {
        const DeepKernel k = deep_kernel(g, B, rf);
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr;
        deep_cfg(cfg, attr, p, 0);
        if (deep_attrs(k, p.smem) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&active, (const void *)k, &cfg) != cudaSuccess || active < 1) {
            cudaGetLastError();
            return 0;
        }
    }
    *out = p;
    return 1;
}

cudaError_t xk_life_step_deep(uint32_t *bits, const LifeGeo &g, uint32_t rule0, uint32_t rule1, int generations,
                              const DeepPlan &p, unsigned int *gave_up, cudaStream_t s)
{
    const DeepKernel k = deep_kernel(g, p.B, xk_rule_form(rule0, rule1));
    if (!k || generations < 1) return cudaErrorInvalidValue;
    cudaError_t e = deep_attrs(k, p.smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    deep_cfg(cfg, attr, p, s);
    return cudaLaunchKernelEx(&cfg, k, bits, g, xk_life_table9(rule0, rule1), generations, p.R, p.bands, gave_up);
}
