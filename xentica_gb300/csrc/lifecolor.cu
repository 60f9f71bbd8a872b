// Life with inherited colour channels (the reference's GameOfLifeColor,
// examples/game_of_life.py:112-159) for sm_103a.
//
// A cell is a uint32 packed LSB first in declaration order
// (properties.py:496-541): state (1 bit) | red << 1 | green << 9 | blue << 17.
// Emit copies every field into every buffer, so a neighbour's buffer is its
// main state: emit is fused away.  Per cell, in the reference's integer
// arithmetic (its absorb as traced):
//   alive  = sum_k state_k
//   state' = ((8 >> alive) & 1) | ((12 >> alive) & 1 & state)
//   c'     = (unsigned char)((sum_k (c_k + 1)) * state')      for c = r, g, b
// and the colour (MovingAverage, color_effects.py:106-130)
//   new = state' * c' * SMOOTH, clamped to [old - FADE_OUT, old + FADE_IN].
// An off-board neighbour of a static border reads as the whole border
// container (border.py:144-151).  The unsigned sums commute, so the
// neighbour order does not matter.
//
// A launch runs T <= 4 generations of tiles in shared memory.  A tile is 128
// cells by 8 R rows read with a halo of one lane's four cells left and right
// and T rows above and below (its inside is exact after T generations; on a
// torus the tile is a window onto the periodic lattice, with a static border
// cells outside hold the border's container after every generation).  Lane l
// holds four consecutive cells of a row, warp w the rows w R .. w R + R - 1;
// a cell is two words of 16-bit sums-to-be (red | blue << 16 and green |
// state << 16: eight 255s fit), so a row's three-cell sums are one addition
// a word and a cell's neighbour sums two more.  Two buffers alternate, one
// barrier a generation.  The colours of a thread's cells stay in its
// registers for the launch; of a generation only the pixels leave the SM, as
// whole words (xk_store_px4).
//
// Colours whose range the host knows to fit 16 bits (it knows the loaded ones'
// and a fade never leaves that range and the cells' own) are faded two
// channels an instruction.
//
// 1920 x 1080, a frame every generation: 7.6 us a generation, 61 warp
// instructions a cell with the tile's halo, against 17.2 us and 250 with one
// launch a generation on plain neighbour loads.  Bound by latency at 16 warps
// an SM (issue 46 %): the load of a tile with its colours, the barriers.
// Measured and not kept: three blocks an SM (80 registers, spills: 9.1 us),
// three generations a launch (10.3 us), loads behind per-row branches (8.5
// us).
#include "xk_internal.cuh"

#include "frame.cuh"

#define XK_LC_WARPS 8
#define XK_LC_MAXT 4

struct LColorParams {
    int32_t W, H;
    int32_t T, TH;              // generations, rows of a tile's inside
    uint32_t border_a, border_b;
    int32_t fade_in, neg_fade_out, smooth;
    uint8_t *frames;            // null, or the W x H RendererPlain frames (zoom 1, no offset)
    int32_t frame_smooth;       // their SMOOTH_FACTOR (0: none)
};

// the two shared words of a packed cell, and back
__device__ __forceinline__ void xk_lc_split(uint32_t w, uint32_t &a, uint32_t &b)
{
    a = (w >> 1) & 0x00FF00FFu;
    b = ((w >> 9) & 0xFFu) | w << 16;
    b &= 0x100FFu;
}

__device__ __forceinline__ uint32_t xk_lc_join(uint32_t a, uint32_t b)
{
    return a << 1 | b >> 16 | (b & 0xFFu) << 9;
}

struct LcRow {
    uint32_t a[4], b[4];
};

// a row's words of this lane, and the sums of each cell with its two
// neighbours in the row (the outer lanes' outer neighbours read as 0: their
// cells are halo)
__device__ __forceinline__ void xk_lc_row(const uint4 *A, const uint4 *B, int at, int lane, LcRow &v, LcRow &h)
{
    const uint4 a = A[at], b = B[at];
    v.a[0] = a.x; v.a[1] = a.y; v.a[2] = a.z; v.a[3] = a.w;
    v.b[0] = b.x; v.b[1] = b.y; v.b[2] = b.z; v.b[3] = b.w;
    const uint32_t la = __shfl_up_sync(0xFFFFFFFFu, a.w, 1), ra = __shfl_down_sync(0xFFFFFFFFu, a.x, 1);
    const uint32_t lb = __shfl_up_sync(0xFFFFFFFFu, b.w, 1), rb = __shfl_down_sync(0xFFFFFFFFu, b.x, 1);
    h.a[0] = la + a.x + a.y; h.a[1] = a.x + a.y + a.z; h.a[2] = a.y + a.z + a.w; h.a[3] = a.z + a.w + ra;
    h.b[0] = lb + b.x + b.y; h.b[1] = b.x + b.y + b.z; h.b[2] = b.y + b.z + b.w; h.b[3] = b.z + b.w + rb;
}

// The colours of a lane's four cells of one row.  Wide: three ints a cell.
// Packed: red | blue << 16 a cell and green of two cells a word, the fades as
// 16-bit pairs: taken when the host knows every colour, and every sum of a
// colour and a fade, to fit 16 bits (xk_lifecolor_packs).
template <bool PACKED>
struct LcColors;

template <>
struct LcColors<false> {
    int c[4][3];
    __device__ __forceinline__ void set(int k, int r, int g, int b)
    {
        c[k][0] = r;
        c[k][1] = g;
        c[k][2] = b;
    }
    __device__ __forceinline__ void get(int k, int *v) const
    {
        v[0] = c[k][0];
        v[1] = c[k][1];
        v[2] = c[k][2];
    }
    __device__ __forceinline__ void fade(const uint32_t *a, const uint32_t *b, const LColorParams &p)
    {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            c[k][0] = xk_fade((int)(a[k] & 0xFFu) * p.smooth, c[k][0], p.fade_in, p.neg_fade_out);
            c[k][1] = xk_fade((int)(b[k] & 0xFFu) * p.smooth, c[k][1], p.fade_in, p.neg_fade_out);
            c[k][2] = xk_fade((int)(a[k] >> 16) * p.smooth, c[k][2], p.fade_in, p.neg_fade_out);
        }
    }
    __device__ __forceinline__ void pixels(uint32_t *w, int frame_smooth) const
    {
        uint32_t px[3][4];
#pragma unroll
        for (int k = 0; k < 12; ++k) {
            const int v = c[k / 3][k % 3];
            px[k % 3][k / 3] = frame_smooth <= 1 && xk_px_small(v) ? (uint32_t)v : xk_pixel(v, frame_smooth);
        }
        xk_pack_px4(px[0], px[1], px[2], w);
    }
};

template <>
struct LcColors<true> {
    uint32_t rb[4], gg[2];
    __device__ __forceinline__ void set(int k, int r, int g, int b)
    {
        rb[k] = __byte_perm((uint32_t)r, (uint32_t)b, 0x5410);
        gg[k >> 1] = k & 1 ? __byte_perm(gg[k >> 1], (uint32_t)g, 0x5410) : (uint32_t)g;
    }
    __device__ __forceinline__ void get(int k, int *v) const
    {
        v[0] = (int16_t)rb[k];
        v[1] = (int16_t)(gg[k >> 1] >> (k & 1 ? 16 : 0));
        v[2] = (int)rb[k] >> 16;
    }
    __device__ __forceinline__ void fade(const uint32_t *a, const uint32_t *b, const LColorParams &p)
    {
        const uint32_t in = (uint32_t)p.fade_in * 0x10001u, out = ((uint32_t)p.neg_fade_out & 0xFFFFu) * 0x10001u;
        auto one = [&](uint32_t v, uint32_t old) {
            return __viaddmax_s16x2(old, out, __viaddmin_s16x2(old, in, v));
        };
#pragma unroll
        for (int k = 0; k < 4; ++k) rb[k] = one(a[k] * (uint32_t)p.smooth, rb[k]);
#pragma unroll
        for (int k = 0; k < 2; ++k)
            gg[k] = one(__byte_perm(b[2 * k], b[2 * k + 1], 0x5410) * (uint32_t)p.smooth, gg[k]);
    }
    __device__ __forceinline__ void pixels(uint32_t *w, int) const
    {
        w[0] = __byte_perm(__byte_perm(rb[0], gg[0], 0x7240), rb[1], 0x4210);
        w[1] = __byte_perm(__byte_perm(gg[0], rb[1], 0x0062), __byte_perm(rb[2], gg[1], 0x0040), 0x5410);
        w[2] = __byte_perm(__byte_perm(rb[2], rb[3], 0x0042), __byte_perm(gg[1], rb[3], 0x0062), 0x5410);
    }
};

// COL: the model's colours (XK_LC_*); FRAME: frames are written
#define XK_LC_NONE 0
#define XK_LC_WIDE 1
#define XK_LC_PACKED 2
template <int R, bool TORUS, int COL, bool FRAME>
__global__ void __launch_bounds__(32 * XK_LC_WARPS, 2)
xk_k_lifecolor(const uint32_t *__restrict__ src, uint32_t *__restrict__ dst, int32_t *__restrict__ col,
               LColorParams p)
{
    extern __shared__ uint4 xk_lc_sm[];                 // [parity][a, b][row][lane]
    constexpr int ROWS = XK_LC_WARPS * R, HALF = ROWS * 32;
    constexpr bool COLOR = COL != XK_LC_NONE;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x0 = blockIdx.x * 120, y0 = blockIdx.y * p.TH, r0 = warp * R;
    // this lane's first cell (compared unsigned: the tiles of the widest rows
    // end beyond 2^31)
    const uint32_t xu = (uint32_t)x0 + 4u * (uint32_t)lane - 4u;
    const int x = (int)xu;
    int xs[4];
    bool xin[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        xin[k] = xu + k < (uint32_t)p.W;
        xs[k] = TORUS && !xin[k] ? xk_wrap_column(xu + k, p.W) : (int)(xu + k);
    }
    // the cells this thread keeps colours of and writes: inside the tile and
    // the lattice
    const bool lin = lane >= 1 && lane <= 30 && xu < (uint32_t)p.W;
    const bool quads = (p.W & 3) == 0;                  // rows start on 16 bytes
    // lanes 1 .. last store whole quads of pixels together
    const int last = min(30, (p.W - x0) >> 2);
    xk_grid_dep_wait();                 // launched as a dependent of the previous launch
    LcColors<COL == XK_LC_PACKED> c[R];
    int ys[R];                                          // the rows read (wrapped, or held to the lattice)
    {
        int yw = y0 - p.T + r0;
        if (TORUS) {
            yw %= p.H;
            if (yw < 0) yw += p.H;
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            ys[i] = TORUS ? yw : min(max(yw, 0), p.H - 1);
            yw = TORUS && yw + 1 == p.H ? 0 : yw + 1;
        }
    }
    auto mine = [&](int i) {                            // row i inside the tile and the lattice
        const int r = r0 + i;
        return r >= p.T && r < p.T + p.TH && y0 - p.T + r < p.H;
    };
    auto put = [&](int i, const uint32_t *w) {
        uint32_t a[4], b[4];
        const int y = y0 - p.T + r0 + i;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            xk_lc_split(w[k], a[k], b[k]);
            if (!TORUS && !(y >= 0 && y < p.H && xin[k])) {
                a[k] = p.border_a;
                b[k] = p.border_b;
            }
        }
        xk_lc_sm[(r0 + i) * 32 + lane] = make_uint4(a[0], a[1], a[2], a[3]);
        xk_lc_sm[HALF + (r0 + i) * 32 + lane] = make_uint4(b[0], b[1], b[2], b[3]);
    };
    if (quads) {
        // no branch between the loads: all of them are in flight at once
        const int xq = TORUS ? xs[0] : min(max(x, 0), p.W - 4);
        uint4 w[R];
#pragma unroll
        for (int i = 0; i < R; ++i) w[i] = __ldg((const uint4 *)(src + (int64_t)ys[i] * p.W + xq));
        if (COLOR) {
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int4 *cp = (const int4 *)(col + 3 * ((int64_t)ys[i] * p.W + xq));
                const bool own = lin && mine(i);
                int4 f[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) f[k] = own ? cp[k] : make_int4(0, 0, 0, 0);
                c[i].set(0, f[0].x, f[0].y, f[0].z);
                c[i].set(1, f[0].w, f[1].x, f[1].y);
                c[i].set(2, f[1].z, f[1].w, f[2].x);
                c[i].set(3, f[2].y, f[2].z, f[2].w);
            }
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const uint32_t v[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
            put(i, v);
        }
    } else {
#pragma unroll
        for (int i = 0; i < R; ++i) {
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                w[k] = __ldg(src + (int64_t)ys[i] * p.W + (TORUS ? xs[k] : min(max(xs[k], 0), p.W - 1)));
            put(i, w);
            if (COLOR) {
                const int32_t *cp = col + 3 * ((int64_t)ys[i] * p.W + x);
                const bool own = lin && mine(i);
                int f[12];
#pragma unroll
                for (int k = 0; k < 12; ++k) f[k] = own && xin[k / 3] ? cp[k] : 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) c[i].set(k, f[3 * k], f[3 * k + 1], f[3 * k + 2]);
            }
        }
    }
    for (int g = 0; g < p.T; ++g) {
        __syncthreads();
        const uint4 *A = xk_lc_sm + (g & 1) * 2 * HALF, *B = A + HALF;
        uint4 *nA = xk_lc_sm + ((g & 1) ^ 1) * 2 * HALF, *nB = nA + HALF;
        const bool end = g + 1 == p.T;
        // rows beyond the tile read as its own: their neighbours are halo
        LcRow v, h, vd, hu, hd;
        xk_lc_row(A, B, max(r0 - 1, 0) * 32 + lane, lane, v, hu);
        xk_lc_row(A, B, r0 * 32 + lane, lane, v, h);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int r = r0 + i, y = y0 - p.T + r;
            xk_lc_row(A, B, min(r + 1, ROWS - 1) * 32 + lane, lane, vd, hd);
            uint32_t a[4], b[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t sa = hu.a[k] + h.a[k] + hd.a[k] - v.a[k];
                const uint32_t sb = hu.b[k] + h.b[k] + hd.b[k] - v.b[k];
                // born with 3, kept with 2: count | state == 3
                const bool live = ((sb | v.b[k]) >> 16) == 3u;
                a[k] = live ? (sa + 0x00080008u) & 0x00FF00FFu : 0u;
                b[k] = live ? ((sb + 8u) & 0xFFu) | 0x10000u : 0u;
            }
            if (COLOR) c[i].fade(a, b, p);
            if (FRAME && mine(i)) {
                uint8_t *at = p.frames + 3 * (((int64_t)g * p.H + y) * p.W + x);
                uint32_t w[3];
                c[i].pixels(w, p.frame_smooth);
                xk_store_px4(at, w, lane, 1, last);
                if (lane == last + 1 && lin)             // a row's last one to three cells
#pragma unroll
                    for (int k = 0; k < 9; ++k)
                        if (xin[k / 3]) at[k] = (uint8_t)(w[k >> 2] >> (8 * (k & 3)));
            }
            if (end) {
                if (mine(i) && lin) {
                    uint32_t *o = dst + (int64_t)y * p.W + x;
                    if (quads) {
                        *(uint4 *)o = make_uint4(xk_lc_join(a[0], b[0]), xk_lc_join(a[1], b[1]),
                                                 xk_lc_join(a[2], b[2]), xk_lc_join(a[3], b[3]));
                    } else {
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (xin[k]) o[k] = xk_lc_join(a[k], b[k]);
                    }
                }
            } else {
                if (!TORUS) {
                    const bool yin = y >= 0 && y < p.H;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (!(yin && xin[k])) {
                            a[k] = p.border_a;
                            b[k] = p.border_b;
                        }
                }
                nA[r * 32 + lane] = make_uint4(a[0], a[1], a[2], a[3]);
                nB[r * 32 + lane] = make_uint4(b[0], b[1], b[2], b[3]);
            }
            hu = h;
            h = hd;
            v = vd;
        }
    }
    if (COLOR && lin) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
            if (!mine(i)) continue;
            int32_t *cp = col + 3 * ((int64_t)ys[i] * p.W + x);
            int f[12];
#pragma unroll
            for (int k = 0; k < 4; ++k) c[i].get(k, f + 3 * k);
            if (quads) {
#pragma unroll
                for (int k = 0; k < 3; ++k) *(int4 *)(cp + 4 * k) = *(const int4 *)(f + 4 * k);
            } else {
#pragma unroll
                for (int k = 0; k < 12; ++k)
                    if (xin[k / 3]) cp[k] = f[k];
            }
        }
    }
}

typedef void (*LcKernel)(const uint32_t *, uint32_t *, int32_t *, LColorParams);

template <int R, bool TORUS>
static LcKernel lc_kernel(int form, bool frames)
{
    if (form == XK_LC_PACKED)
        return frames ? xk_k_lifecolor<R, TORUS, XK_LC_PACKED, true> : xk_k_lifecolor<R, TORUS, XK_LC_PACKED, false>;
    return nullptr;
}

// the forms without packed colours run tiles of 32 rows only
template <bool TORUS>
static LcKernel lc_kernel_4(int form, bool frames)
{
    if (form == XK_LC_NONE) return xk_k_lifecolor<4, TORUS, XK_LC_NONE, false>;
    if (form == XK_LC_WIDE)
        return frames ? xk_k_lifecolor<4, TORUS, XK_LC_WIDE, true> : xk_k_lifecolor<4, TORUS, XK_LC_WIDE, false>;
    return lc_kernel<4, TORUS>(form, frames);
}

static LcKernel lc_pick(int R, bool torus, int form, bool frames)
{
    switch (R) {
    case 2: return torus ? lc_kernel<2, true>(form, frames) : lc_kernel<2, false>(form, frames);
    case 5: return torus ? lc_kernel<5, true>(form, frames) : lc_kernel<5, false>(form, frames);
    default: return torus ? lc_kernel_4<true>(form, frames) : lc_kernel_4<false>(form, frames);
    }
}

int xk_lifecolor_max_generations() { return XK_LC_MAXT; }

// A faded colour lies between the old one and the cell's own (0 .. 255
// smooth), so colours never leave the range of the loaded ones and those:
// where that range and a fade on top of it fit 16 bits, they are packed.
static bool lc_packs(const xk_desc &d, const int32_t range[2], const uint8_t *frames, int frame_smooth)
{
    const int64_t lim = 16000;
    return range[0] >= -lim && range[1] <= lim && d.fade_in >= 0 && d.fade_in <= lim && d.fade_out >= 0 &&
           d.fade_out <= lim && d.smooth >= 0 && 255ll * d.smooth <= lim && (!frames || frame_smooth <= 1);
}

cudaError_t xk_lifecolor_step(const uint32_t *src, uint32_t *dst, int32_t *col, const xk_desc &d, int generations,
                              const int32_t color_range[2], cudaStream_t s, uint8_t *frames, int frame_smooth)
{
    if (generations < 1 || generations > XK_LC_MAXT) return cudaErrorInvalidValue;
    LColorParams p;
    p.W = (int32_t)d.size[0];
    p.H = (int32_t)d.size[1];
    p.T = generations;
    const uint32_t border = (uint32_t)d.border_value;
    p.border_a = (border >> 1) & 0x00FF00FFu;
    p.border_b = ((border >> 9) & 0xFFu) | (border & 1u) << 16;
    p.fade_in = d.fade_in;
    p.neg_fade_out = (int32_t)(0u - (uint32_t)d.fade_out);
    p.smooth = d.smooth;
    p.frames = frames;
    p.frame_smooth = frame_smooth;
    const int form = d.color_kind == XK_COLOR_NONE ? XK_LC_NONE
                     : lc_packs(d, color_range, frames, frame_smooth) ? XK_LC_PACKED : XK_LC_WIDE;
    const int64_t gx = ((int64_t)p.W + 119) / 120;
    auto tiles = [&](int R) {
        const int th = XK_LC_WARPS * R - 2 * p.T;
        return gx * (((int64_t)p.H + th - 1) / th);
    };
    // Rows a warp: of 5 and 4, the one whose waves of two blocks an SM cover
    // fewer rows; 2 where tiles of 4 would leave SMs without one (shorter
    // generations, more halo).
    const int64_t sms = xk_sm_count() > 0 ? xk_sm_count() : 1;
    auto waves = [&](int R) { return (tiles(R) + 2 * sms - 1) / (2 * sms) * R; };
    int R = 4;
    if (form == XK_LC_PACKED) R = tiles(4) < sms ? 2 : waves(5) < waves(4) ? 5 : 4;
    p.TH = XK_LC_WARPS * R - 2 * p.T;
    const dim3 grid((unsigned)gx, (unsigned)((p.H + p.TH - 1) / p.TH));
    if (grid.y > 65535u) return cudaErrorInvalidValue;
    const LcKernel k = lc_pick(R, d.torus != 0, form, frames != nullptr);
    const int smem = 4 * XK_LC_WARPS * R * 32 * (int)sizeof(uint4);
    cudaError_t e = xk_smem_attr_at_least((const void *)k, smem);
    if (e != cudaSuccess) return e;
    return xk_launch_pdl(k, grid, dim3(32 * XK_LC_WARPS), (size_t)smem, s, src, dst, col, p);
}
