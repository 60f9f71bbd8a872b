// Life-like generations of lattices that are not 2-D Moore ones (any
// dimensionality, any neighbourhood with offsets of at most one cell per
// axis), bit-packed along axis 0: row r = (x1, x2, ...) with axis 1 fastest,
// 32 cells a word, the 2-D packing of life.cu with n / W rows.
//
// A thread computes one word: the neighbours fall into rows (one per distinct
// offset along the axes above 0); of each row it loads the word and, where
// cells left or right of it are neighbours, the words beside it, and the row's
// one to three shifted words go into a bit-sliced count.  The count's planes
// and the cells select the rule bit through a multiplexer tree over
// warp-uniform masks, as in life_word.cuh.
//
// The six faces of a 3-D lattice have kernels of their own (life.cu,
// life3d_cluster.cu): 100 generations of 128^3 450 -> 169 us.
//
// Bound by instruction issue: a word of 3-D Moore takes 1 073 instructions (its
// 27 row words with their addresses and borders, the count, the rule's 63
// selections), 1.9 us of issue on 152 SMs for the 65 536 words of 128^3, whose
// 2 048 warps fill 58 % of the slots: 3.7 to 4 us a generation, where the
// kernel of the six faces takes 1.6 in a launch of the same size.  100
// generations of 128^3 Moore and the read after them: 425 us, against 18 468 us
// with the byte-per-cell kernel (xk_k_life_nd: one thread a
// cell, 27 loads with 64-bit coordinates), which is left for lattices this
// packing cannot index.
#include <string.h>

#include "life_word.cuh"

namespace {

struct Fa {
    uint32_t s, c;
};

__device__ __forceinline__ Fa fa(uint32_t a, uint32_t b, uint32_t c)
{
    return Fa{xk_lop3_xor3(a, b, c), xk_maj(a, b, c)};
}

// rule bit of 32 cells from the NB planes of the neighbour count and the cells
template <int NB>
__device__ __forceinline__ uint32_t rule_nd(const LifeTable32 &t, const uint32_t *b, uint32_t C)
{
    uint32_t m[1 << NB];     // level 1: dead pairs, then live pairs
#pragma unroll
    for (int q = 0; q < (1 << (NB - 1)); ++q) {
        m[q] = xk_imux(b[0], t.a[q], t.k[q]);
        m[q + (1 << (NB - 1))] = xk_imux(b[0], t.a[16 + q], t.k[16 + q]);
    }
#pragma unroll
    for (int lev = 1; lev < NB; ++lev)
#pragma unroll
        for (int q = 0; q < (1 << (NB - lev)); ++q) m[q] = xk_mux(b[lev], m[2 * q], m[2 * q + 1]);
    return xk_mux(C, m[0], m[1]);
}

// position of a thread's word: row coordinates are up to the caller
struct WordPos {
    uint32_t r;              // row
    int j, jl, jr;           // word and the words beside it (wrapped)
    int lshift, top, use_le, use_re;
};

__device__ __forceinline__ WordPos word_pos(uint32_t idx, const BitsNdGeo &g)
{
    WordPos p;
    p.r = xk_divu(idx, (uint32_t)g.wpr, g.div_wpr);
    p.j = (int)(idx - p.r * (uint32_t)g.wpr);
    const int last = g.wpr - 1;
    p.jl = p.j > 0 ? p.j - 1 : last;
    p.jr = p.j < last ? p.j + 1 : 0;
    p.lshift = p.j > 0 ? 31 : g.rlast - 1;
    p.top = p.j == last ? g.rlast - 1 : 31;
    p.use_le = !g.torus && p.j == 0;
    p.use_re = !g.torus && p.j == last;
    return p;
}

__device__ __forceinline__ RowVec row_vec(const uint32_t *__restrict__ row, const WordPos &p, uint32_t edge)
{
    return xk_row_vec(__ldg(row + p.j), __ldg(row + p.jl), __ldg(row + p.jr), p.lshift, p.top, edge, edge,
                      p.use_le, p.use_re);
}

}  // namespace

// The reference's 3-D Moore neighbourhood (neighborhood.py:151-167: every offset
// but the last, so the cell itself is one of the 26 and (1, 1, 1) is not):
// nine rows, each reduced to a sum and a carry word as it arrives, the rest
// of the count in a carry-save tree
template <bool TORUS>
__global__ void __launch_bounds__(128)
xk_k_life3d_moore(const uint32_t *__restrict__ src, uint32_t *__restrict__ dst, BitsNdGeo g, LifeTable32 t)
{
    const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= g.words) return;
    xk_grid_dep_wait();       // launched as a dependent of the previous generation
    const WordPos p = word_pos(idx, g);
    const uint32_t H = (uint32_t)g.size[1], D = (uint32_t)g.size[2];
    const uint32_t z = xk_divu(p.r, H, g.div_h), y = p.r - z * H;
    const uint32_t ys[3] = {y > 0 ? y - 1 : H - 1, y, y + 1 < H ? y + 1 : 0};
    const uint32_t zs[3] = {z > 0 ? z - 1 : D - 1, z, z + 1 < D ? z + 1 : 0};
    const bool yoff[3] = {!TORUS && y == 0, false, !TORUS && y + 1 == H};
    const bool zoff[3] = {!TORUS && z == 0, false, !TORUS && z + 1 == D};
    const uint32_t edge = g.bfill & 1u;
    uint32_t C = 0;
    Fa f[9];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const int k = 3 * a + b;
            if (!TORUS && (zoff[a] || yoff[b])) {
                f[k] = Fa{k == 8 ? 0u : g.bfill, g.bfill};
                continue;
            }
            const RowVec v = row_vec(src + (zs[a] * H + ys[b]) * (uint32_t)g.wpr, p, edge);
            if (k == 4) C = v.C;
            f[k] = k == 8 ? Fa{v.L ^ v.C, v.L & v.C} : fa(v.L, v.C, v.R);
        }
    uint32_t n[5];
    const Fa s0 = fa(f[0].s, f[1].s, f[2].s), s1 = fa(f[3].s, f[4].s, f[5].s), s2 = fa(f[6].s, f[7].s, f[8].s);
    const Fa s3 = fa(s0.s, s1.s, s2.s);
    n[0] = s3.s;
    // weight 2: nine carries of the rows, s0.c, s1.c, s2.c, s3.c
    const Fa d0 = fa(f[0].c, f[1].c, f[2].c), d1 = fa(f[3].c, f[4].c, f[5].c), d2 = fa(f[6].c, f[7].c, f[8].c);
    const Fa d3 = fa(s0.c, s1.c, s2.c);
    const Fa d4 = fa(d0.s, d1.s, d2.s), d5 = fa(d3.s, d4.s, s3.c);
    n[1] = d5.s;
    // weight 4: d0..d5 carries
    const Fa e0 = fa(d0.c, d1.c, d2.c), e1 = fa(d3.c, d4.c, d5.c);
    n[2] = e0.s ^ e1.s;
    const Fa h = fa(e0.c, e1.c, e0.s & e1.s);      // weight 8
    n[3] = h.s;
    n[4] = h.c;
    uint32_t out = rule_nd<5>(t, n, C);
    if (p.j == g.wpr - 1) out &= g.lastmask;
    dst[idx] = out;
}

// any other neighbourhood: the rows one after another, added to the count's
// planes by ripple
template <int NB>
__global__ void __launch_bounds__(128)
xk_k_life_bits_nd(const uint32_t *__restrict__ src, uint32_t *__restrict__ dst, BitsNdGeo g, LifeTable32 t)
{
    const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= g.words) return;
    xk_grid_dep_wait();       // launched as a dependent of the previous generation
    const WordPos p = word_pos(idx, g);
    int32_t x[XK_MAXDIM];
    {
        uint32_t rest = p.r;
        for (int d = 1; d < g.ndim; ++d) {
            const uint32_t q = d + 1 < g.ndim ? rest / (uint32_t)g.size[d] : 0u;
            x[d] = (int32_t)(rest - q * (uint32_t)g.size[d]);
            rest = q;
        }
    }
    const uint32_t edge = g.bfill & 1u;
    uint32_t n[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) n[b] = 0;
    for (int k = 0; k < g.groups; ++k) {
        int64_t r = 0, stride = 1;
        bool off = false;
        for (int d = 1; d < g.ndim; ++d) {
            int32_t c = x[d] + g.delta[k][d];
            if (c < 0) {
                c += g.size[d];
                off = true;
            } else if (c >= g.size[d]) {
                c -= g.size[d];
                off = true;
            }
            r += c * stride;
            stride *= g.size[d];
        }
        RowVec v;
        if (off && !g.torus) v.L = v.C = v.R = g.bfill;
        else v = row_vec(src + r * g.wpr, p, edge);
        const int has = g.delta[k][0];           // bit 0: left, 1: the cell above, 2: right
        uint32_t add = has & 1 ? v.L : 0u, carry;
        const Fa f = fa(add, has & 2 ? v.C : 0u, has & 4 ? v.R : 0u);
        // the row's sum at weight 1, its carry at weight 2
        add = f.s;
        carry = n[0] & add;
        n[0] ^= add;
        const Fa w = fa(n[1], f.c, carry);
        n[1] = w.s;
        carry = w.c;
#pragma unroll
        for (int b = 2; b < NB; ++b) {
            const uint32_t c = n[b] & carry;
            n[b] ^= carry;
            carry = c;
        }
    }
    const uint32_t C = __ldg(src + idx);
    uint32_t out = rule_nd<NB>(t, n, C);
    if (p.j == g.wpr - 1) out &= g.lastmask;
    dst[idx] = out;
}

int xk_bits_nd_geo(const NdGeo &nd, BitsNdGeo *out)
{
    BitsNdGeo g;
    memset(&g, 0, sizeof(g));
    if (nd.ndim < 1 || nd.nbr < 1 || nd.nbr > 31) return 0;
    g.ndim = nd.ndim;
    int64_t rows = 1;
    for (int d = 0; d < nd.ndim; ++d) {
        if (nd.size[d] > 0x7FFFFFFFll) return 0;
        g.size[d] = (int32_t)nd.size[d];
        if (d > 0) rows *= nd.size[d];
        if (rows > 0x7FFFFFFFll) return 0;
    }
    const LifeGeo lg = xk_life_geo(nd.size[0], rows, nd.torus, (int)nd.border_state);
    // 32-bit word indices, and so 32-bit grids, in the kernels
    if (rows * lg.wpr > 0x7FFFFFFFll) return 0;
    g.wpr = lg.wpr;
    g.rlast = lg.rlast;
    g.lastmask = lg.lastmask;
    g.torus = lg.torus;
    g.bfill = lg.bfill;
    g.div_wpr = lg.div_wpr;
    g.words = (uint32_t)(rows * lg.wpr);
    g.div_h = nd.ndim == 3 ? xk_div_magic((uint64_t)nd.size[1], (uint64_t)rows) : 0u;
    // neighbours by row; delta[k][0] of a row: which of left, above, right it has
    for (int k = 0; k < nd.nbr; ++k) {
        for (int d = 0; d < nd.ndim; ++d)
            if (nd.delta[k][d] < -1 || nd.delta[k][d] > 1) return 0;
        int at = 0;
        for (; at < g.groups; ++at) {
            bool same = true;
            for (int d = 1; d < nd.ndim; ++d) same = same && g.delta[at][d] == nd.delta[k][d];
            if (same) break;
        }
        if (at == g.groups) {
            for (int d = 1; d < nd.ndim; ++d) g.delta[at][d] = nd.delta[k][d];
            ++g.groups;
        }
        const int bit = 1 << (nd.delta[k][0] + 1);
        if (g.delta[at][0] & bit) return 0;                 // a neighbour twice
        g.delta[at][0] = (int8_t)(g.delta[at][0] | bit);
    }
    g.nbr = nd.nbr;
    // the six faces, in any order
    g.faces3d = nd.ndim == 3 && nd.nbr == 6;
    for (int k = 0; k < nd.nbr && g.faces3d; ++k)
        g.faces3d = abs(nd.delta[k][0]) + abs(nd.delta[k][1]) + abs(nd.delta[k][2]) == 1;
    // 26 of the 27 offsets, (1, 1, 1) the one left out
    g.moore3d = 0;
    if (nd.ndim == 3 && nd.nbr == 26) {
        for (int k = 0; k < g.groups; ++k)
            if (g.delta[k][1] == 1 && g.delta[k][2] == 1) g.moore3d = g.delta[k][0] == 3;
    }
    *out = g;
    return 1;
}

cudaError_t xk_life_step_bits_nd(const uint32_t *src, uint32_t *dst, const BitsNdGeo &g, uint32_t rule0,
                                 uint32_t rule1, cudaStream_t s)
{
    LifeTable32 t;
    auto mask = [](uint32_t r, int n) { return 0u - ((r >> n) & 1u); };
    for (int q = 0; q < 32; ++q) {
        const uint32_t r = q < 16 ? rule0 : rule1;
        const int n = 2 * (q & 15);
        t.a[q] = mask(r, n);
        t.k[q] = xk_mux_coef(mask(r, n), mask(r, n + 1));
    }
    const int threads = 128;
    const dim3 grid((g.words + threads - 1) / threads), block(threads);
    if (g.moore3d)
        return g.torus ? xk_launch_pdl(xk_k_life3d_moore<true>, grid, block, 0, s, src, dst, g, t)
                       : xk_launch_pdl(xk_k_life3d_moore<false>, grid, block, 0, s, src, dst, g, t);
    // planes of a count of up to nbr neighbours
    if (g.nbr <= 7) return xk_launch_pdl(xk_k_life_bits_nd<3>, grid, block, 0, s, src, dst, g, t);
    if (g.nbr <= 15) return xk_launch_pdl(xk_k_life_bits_nd<4>, grid, block, 0, s, src, dst, g, t);
    return xk_launch_pdl(xk_k_life_bits_nd<5>, grid, block, 0, s, src, dst, g, t);
}
