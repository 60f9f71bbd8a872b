// Temporally blocked Life-like generations for 2-D lattices too large for one
// CTA: T generations per launch (T <= XK_TB_MAXT), each CTA on a tile of its
// own in registers.
//
// Tile: 32 words (1024 cells) by 8 B rows, read from the lattice with a halo
// -- one word left and right, T rows above and below -- so the interior
// (words 1..30, rows T..T + TH - 1 with TH = 8 B - 2 T) is exact after T
// generations: a cell's value after k generations depends only on cells
// within k of it, and the halo is T >= k cells deep in rows and 32 cells deep
// in columns.  Tile cell b of word w is the lattice cell x0 - 32 + 32 w + b of
// row y0 - T + r; on a torus that coordinate is taken modulo W and H (the
// tile is a window onto the periodic lattice, so a word may straddle the
// wrap), with a static border cells outside the lattice hold the border state
// and are reset to it after every generation.
//
// Each of the 8 warps owns a band of B tile rows, lane w holding word w of
// every row in registers for the whole launch; a generation walks down the
// band with the column sums (s, c) = FA(L, C, R) of the rows above, at and
// below, the left and right neighbour bits from the adjacent lanes by
// shuffles.  Only the band's first and last row go through shared memory, for
// the bands beside it: two words a lane, double-buffered by generation, one
// barrier each.  Lanes 0 and 31 and the rows outside the interior compute on
// incomplete neighbourhoods; their values are never stored.
//
// Bound by the logic pipe (63 %; 39 instructions a word, of which a rule read
// from a table is 18) and by about 3 us a launch (its start, the tile's loads
// and stores).  4096 x 4096, such a rule, 960 generations: 1 295 us with 12
// generations a launch and tiles of 21 rows a warp (145 of the 152 SMs hold
// one; 1 310 with 16 generations), 1 414 with 8, 1 605 with 8 on tiles of 12
// rows a warp (two on most SMs, one on the others); twice that with the tile
// in shared memory (every word of every generation loaded, stored and waited
// for).
//
// Requires W >= 64 (a 32-cell window wraps at most once).
#include <string.h>

#include "life_word.cuh"

#define XK_TB_MAXT XK_TB_DEEPEST
#define XK_TB_WARPS 8

struct TbParams {
    LifeGeo g;
    int32_t T, TH;             // generations, interior rows
};

// column sums of a row's word: the cells left and right come from the lanes
// beside this one (lanes 0 and 31 read bits of lanes they are not next to:
// halo cells)
__device__ __forceinline__ void xk_tb_sums(uint32_t c, uint32_t &s, uint32_t &cy)
{
    const uint32_t l = __shfl_up_sync(0xFFFFFFFFu, c, 1), r = __shfl_down_sync(0xFFFFFFFFu, c, 1);
    const uint32_t L = __funnelshift_l(l, c, 1), R = __funnelshift_r(c, r, 1);
    s = xk_lop3_xor3(L, c, R);
    cy = xk_maj(L, c, R);
}

template <int B, bool TORUS, int RF>
__global__ void __launch_bounds__(32 * XK_TB_WARPS)
xk_k_life_tb(const uint32_t *__restrict__ src, uint32_t *__restrict__ dst, TbParams p, LifeTable9 t9)
{
    const auto &t = RuleForm<RF>::make(t9);
    constexpr int ROWS = B * XK_TB_WARPS;
    // [parity][warp, and one either side][first, last row][lane]
    __shared__ uint32_t edge[2][XK_TB_WARPS + 2][2][32];
    const LifeGeo &g = p.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x0 = blockIdx.x * 30 * 32;                   // first interior cell
    const int y0 = blockIdx.y * p.TH;                      // first interior row
    const int X = x0 - 32 + 32 * lane;                     // this lane's first cell
    const int r0 = warp * B;
    // bits of this lane's word outside the lattice (static border only)
    uint32_t outside = 0;
    if (!TORUS) {
        if (X < 0 || X >= g.W) outside = 0xFFFFFFFFu;
        else if (g.W - X < 32) outside = ~((1u << (g.W - X)) - 1u);
    }
    // the 32 cells from X: bits sh.. of word jw and the next word's (padding
    // bits are 0), and past the row's end its first cells (W >= 64: word 0
    // holds 32 of them)
    int xm = X;
    if (TORUS) {
        xm %= g.W;
        if (xm < 0) xm += g.W;
    } else if (xm < 0 || xm >= g.W) {
        xm = 0;                                            // outside: replaced below
    }
    const int jw = xm >> 5, sh = xm & 31, avail = g.W - xm;
    const bool two = jw + 1 < g.wpr, wraps = TORUS && avail < 32;
    int yr = y0 - p.T + r0;                                // this warp's first row
    int ym = yr;
    if (TORUS) {
        ym %= g.H;
        if (ym < 0) ym += g.H;
    }
    xk_grid_dep_wait();       // launched as a dependent of the previous launch
    uint32_t w[B];
#pragma unroll
    for (int i = 0; i < B; ++i) {
        const uint32_t *row = src + (int64_t)(TORUS ? ym : min(max(yr + i, 0), g.H - 1)) * g.wpr;
        const uint32_t a = __ldg(row + jw), b = two ? __ldg(row + jw + 1) : 0u;
        const uint32_t c = wraps ? __ldg(row) << avail : 0u;
        w[i] = __funnelshift_r(a, b, sh) | c;
        ym = ym + 1 == g.H ? 0 : ym + 1;
        if (!TORUS) {
            const bool off = yr + i < 0 || yr + i >= g.H;
            w[i] = off ? g.bfill : (w[i] & ~outside) | (g.bfill & outside);
        }
    }
    for (int gen = 0; gen < p.T; ++gen) {
        uint32_t (*e)[2][32] = edge[gen & 1];
        e[warp + 1][0][lane] = w[0];
        e[warp + 1][1][lane] = w[B - 1];
        __syncthreads();
        // rows beyond the tile (warp 0's above, the last one's below) read
        // whatever is there: their neighbours are halo
        uint32_t su, cu, sm, cm, sd, cd;
        xk_tb_sums(e[warp][1][lane], su, cu);
        const uint32_t below = e[warp + 2][0][lane];
        xk_tb_sums(w[0], sm, cm);
#pragma unroll
        for (int i = 0; i < B; ++i) {
            const uint32_t c = w[i];
            xk_tb_sums(i + 1 < B ? w[i + 1 < B ? i + 1 : i] : below, sd, cd);
            uint32_t out = xk_life_word9(su, cu, sm, cm, sd, cd, c, t);
            if (!TORUS) {
                const bool off = yr + i < 0 || yr + i >= g.H;
                out = off ? g.bfill : (out & ~outside) | (g.bfill & outside);
            }
            w[i] = out;
            su = sm;
            cu = cm;
            sm = sd;
            cm = cd;
        }
    }
    // the interior: lanes 1..30, rows T .. T + TH - 1, where they are cells
    const int j = (x0 >> 5) + lane - 1;
    if (lane < 1 || lane > 30 || j >= g.wpr) return;
#pragma unroll
    for (int i = 0; i < B; ++i) {
        const int r = r0 + i, y = yr + i;
        if (r >= p.T && r < p.T + p.TH && y < g.H)
            dst[(int64_t)y * g.wpr + j] = j == g.wpr - 1 ? w[i] & g.lastmask : w[i];
    }
}

int xk_life_tb_supported(const LifeGeo &g) { return g.W >= 64; }

typedef void (*TbKernel)(const uint32_t *, uint32_t *, TbParams, LifeTable9);

template <int B>
static TbKernel tb_kernel(bool torus, bool conway)
{
    if (torus) return conway ? xk_k_life_tb<B, true, XK_RULE_CONWAY> : xk_k_life_tb<B, true, XK_RULE_TABLE>;
    return conway ? xk_k_life_tb<B, false, XK_RULE_CONWAY> : xk_k_life_tb<B, false, XK_RULE_TABLE>;
}

cudaError_t xk_life_step_tb(const uint32_t *src, uint32_t *dst, const LifeGeo &g, const LifeTable9 &t,
                            int T, cudaStream_t s)
{
    if (T < 1 || T > XK_TB_MAXT || g.W < 64) return cudaErrorInvalidValue;
    // Rows a warp: the height whose tiles, dealt to the SMs, leave the
    // fewest rows on the fullest one (ties: the taller, less halo).
    const int64_t gx = (g.W + 30 * 32 - 1) / (30 * 32), sms = xk_sm_count() > 0 ? xk_sm_count() : 1;
    // Against heights of 16, 12, 8 and 4 alone, 12 generations of lattices
    // with sides up to 4000 and at least 2^20 cells take 22 % fewer rows.
    static const int heights[] = {21, 17, 14, 12, 10, 8, 7, 6, 5, 4};
    int B = 0;
    int64_t best = 0;
    for (int b : heights) {
        const int th = XK_TB_WARPS * b - 2 * T;
        if (th <= 0) continue;
        const int64_t tiles = gx * ((g.H + th - 1) / th), rows = (tiles + sms - 1) / sms * XK_TB_WARPS * b;
        if (!B || rows < best) {
            B = b;
            best = rows;
        }
    }
    TbParams p;
    p.g = g;
    p.T = T;
    p.TH = XK_TB_WARPS * B - 2 * T;
    const dim3 grid((unsigned)gx, (unsigned)((g.H + p.TH - 1) / p.TH));
    if (grid.y > 65535u) return cudaErrorInvalidValue;
    // B3/S23 runs the instantiation with the rule compiled in
    const LifeTable9 table = xk_life_table9(8u, 12u);
    const bool conway = memcmp(&t, &table, sizeof(t)) == 0, torus = g.torus != 0;
    TbKernel k = nullptr;
    switch (B) {
    case 4: k = tb_kernel<4>(torus, conway); break;
    case 5: k = tb_kernel<5>(torus, conway); break;
    case 6: k = tb_kernel<6>(torus, conway); break;
    case 7: k = tb_kernel<7>(torus, conway); break;
    case 8: k = tb_kernel<8>(torus, conway); break;
    case 10: k = tb_kernel<10>(torus, conway); break;
    case 12: k = tb_kernel<12>(torus, conway); break;
    case 14: k = tb_kernel<14>(torus, conway); break;
    case 17: k = tb_kernel<17>(torus, conway); break;
    default: k = tb_kernel<21>(torus, conway); break;
    }
    return xk_launch_pdl(k, grid, dim3(32 * XK_TB_WARPS), 0, s, src, dst, p, t);
}
