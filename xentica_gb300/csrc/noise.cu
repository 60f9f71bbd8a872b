// Per-cell noise (the reference's NoiseTV, examples/noisetv.py:13-31) for
// sm_103a.
//
// A cell is one RandomProperty (uint16).  Emit writes nothing; absorb reads
// the property once and the colour reads its uniform draw, each read one
// advance of x = (x * 58321 + 11113) % 65535 (properties.py:638-660); the
// colour is (unsigned)((float)x / 65535 * 255) on every channel, through
// MovingAverage (color_effects.py:106-130), and the cell stores x.  No cell
// reads another, so one launch runs many generations of a cell in registers,
// with or without a frame for each: its state and colour are read once and
// written once, and of a generation only the pixels leave the SM.
//
// A thread owns four consecutive cells: their pixels are three whole words of
// a frame (xk_store_px4).  The two advances of a generation are one composed
// map x -> (a x + c) % 65535 (a, c below 65535, so a x + c stays below
// 2^32 - 1), the remainder folded from the halves (2^16 = 1 mod 65535); the
// grey level is x * 65281 >> 24, equal to the float expression for every
// x < 65535 (tests/test_noise_cpu.py).  A cell whose three colours are equal
// keeps them equal: one channel is computed for it.
//
// Bound by instruction issue without frames, by the frames' writes with them.
// 1920 x 1080, a frame every generation: one launch a generation took 9.8 us
// (state, colours and frame through L2, 26.8 warp instructions a cell), now 1.8.
// (Measured and not kept: the grey level of every x from a 65 535-byte table,
// which put a load in each generation's dependent chain.)
#include "xk_internal.cuh"

#include "frame.cuh"

struct NoiseParams {
    int64_t n;
    int32_t color_kind;          // XK_COLOR_*
    int32_t fade_in, neg_fade_out, smooth;
    int32_t generations;         // generations per launch
    uint8_t *frames;             // the zoom-1 RendererPlain frames of a 2-D lattice, 3 n bytes each
    int32_t frame_smooth;        // their SMOOTH_FACTOR (0: none)
    int32_t small;               // xk_px_stays_small
};

// the two advances of a generation composed: 58321^2 and 58321 * 11113 + 11113, mod 65535
#define XK_NOISE_A2 ((58321ull * 58321ull) % 65535ull)
#define XK_NOISE_C2 ((58321ull * 11113ull + 11113ull) % 65535ull)

__device__ __forceinline__ uint32_t xk_noise_advance(uint32_t x)
{
    const uint32_t t = (uint32_t)XK_NOISE_A2 * x + (uint32_t)XK_NOISE_C2;
    const uint32_t s = t - 65535u * (t >> 16);           // low half + high half, at most 131069
    return __viaddmin_u32(s, 0u - 65535u, s);            // s - 65535 where that does not wrap
}

__device__ __forceinline__ int xk_noise_grey(uint32_t x) { return (int)((x * 65281u) >> 24); }

// the generations of a thread's four cells; CH: colour channels computed (1:
// all equal); SMALL: a pixel is its colour's low byte
template <bool FRAME, int CH, bool SMALL>
__device__ __forceinline__ void xk_noise_cells(uint32_t x[4], int c[4][3], const NoiseParams &p, int64_t i,
                                               int lane, bool whole_warp)
{
    uint8_t *px = FRAME ? p.frames + 3 * i : nullptr;
    for (int g = 0; g < p.generations; ++g) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            x[k] = xk_noise_advance(x[k]);
            const int v = xk_noise_grey(x[k]) * p.smooth;
#pragma unroll
            for (int ch = 0; ch < CH; ++ch) c[k][ch] = xk_fade(v, c[k][ch], p.fade_in, p.neg_fade_out);
        }
        if (FRAME) {
            uint32_t r[3][4], w[3];
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int ch = 0; ch < 3; ++ch)
                    r[ch][k] = ch >= CH ? r[0][k] : SMALL ? (uint32_t)c[k][ch] : xk_pixel(c[k][ch], p.frame_smooth);
            if (whole_warp) {
                xk_pack_px4(r[0], r[1], r[2], w);
                xk_store_px4(px, w, lane, 0, 31);
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (i + k < p.n)
                        for (int ch = 0; ch < 3; ++ch) px[3 * k + ch] = (uint8_t)r[ch][k];
            }
            px += 3 * p.n;
        }
    }
    if (CH == 1) {
#pragma unroll
        for (int k = 0; k < 4; ++k) c[k][1] = c[k][2] = c[k][0];
    }
}

template <bool FRAME>
__global__ void __launch_bounds__(256)
xk_k_noise(uint16_t *__restrict__ cells, int32_t *__restrict__ col, NoiseParams p)
{
    const int64_t i = 4 * ((int64_t)blockIdx.x * blockDim.x + threadIdx.x);
    const int lane = threadIdx.x & 31;
    const bool whole_warp = i - 4 * lane + 128 <= p.n;
    xk_grid_dep_wait();                 // launched as a dependent of the previous launch
    if (i >= p.n) return;               // never in a whole warp
    const bool ma = p.color_kind != XK_COLOR_NONE;
    uint32_t x[4] = {0, 0, 0, 0};
    int c[4][3] = {};
    if (i + 4 <= p.n) {
        const uint2 v = *(const uint2 *)(cells + i);      // rows of the device buffers start aligned
        x[0] = v.x & 0xFFFFu;
        x[1] = v.x >> 16;
        x[2] = v.y & 0xFFFFu;
        x[3] = v.y >> 16;
        if (ma) {
            int f[12];
#pragma unroll
            for (int k = 0; k < 3; ++k) *(int4 *)(f + 4 * k) = *(const int4 *)(col + 3 * i + 4 * k);
#pragma unroll
            for (int k = 0; k < 12; ++k) c[k / 3][k % 3] = f[k];
        }
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (i + k < p.n) {
                x[k] = cells[i + k];
                if (ma)
                    for (int ch = 0; ch < 3; ++ch) c[k][ch] = col[3 * (i + k) + ch];
            }
    }
    if (ma) {
        bool grey = true, small = p.small != 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            grey = grey && c[k][0] == c[k][1] && c[k][0] == c[k][2];
            small = small && xk_px_small(c[k][0]) && xk_px_small(c[k][1]) && xk_px_small(c[k][2]);
        }
        // one form for a whole warp: its frame stores are the warp's
        if (whole_warp) {
            grey = __all_sync(0xFFFFFFFFu, grey);
            small = __all_sync(0xFFFFFFFFu, small);
        }
        if (!FRAME || !small) {
            if (!FRAME && grey) xk_noise_cells<FRAME, 1, false>(x, c, p, i, lane, whole_warp);
            else xk_noise_cells<FRAME, 3, false>(x, c, p, i, lane, whole_warp);
        } else {
            if (grey) xk_noise_cells<FRAME, 1, true>(x, c, p, i, lane, whole_warp);
            else xk_noise_cells<FRAME, 3, true>(x, c, p, i, lane, whole_warp);
        }
    } else {
        for (int g = 0; g < p.generations; ++g)
#pragma unroll
            for (int k = 0; k < 4; ++k) x[k] = xk_noise_advance(x[k]);
    }
    if (i + 4 <= p.n) {
        *(uint2 *)(cells + i) = make_uint2(x[0] | x[1] << 16, x[2] | x[3] << 16);
        if (ma) {
            int f[12];
#pragma unroll
            for (int k = 0; k < 12; ++k) f[k] = c[k / 3][k % 3];
#pragma unroll
            for (int k = 0; k < 3; ++k) *(int4 *)(col + 3 * i + 4 * k) = *(const int4 *)(f + 4 * k);
        }
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (i + k < p.n) {
                cells[i + k] = (uint16_t)x[k];
                if (ma)
                    for (int ch = 0; ch < 3; ++ch) col[3 * (i + k) + ch] = c[k][ch];
            }
    }
}

cudaError_t xk_noise_step(uint16_t *cells, int32_t *col, const xk_desc &d, int64_t n, int generations,
                          cudaStream_t s, uint8_t *frames, int frame_smooth)
{
    if (generations < 1) return cudaErrorInvalidValue;
    NoiseParams p;
    p.n = n;
    p.color_kind = d.color_kind;
    p.fade_in = d.fade_in;
    p.neg_fade_out = (int32_t)(0u - (uint32_t)d.fade_out);
    p.smooth = d.smooth;
    p.generations = generations;
    p.frames = frames;
    p.frame_smooth = frame_smooth;
    p.small = xk_px_stays_small(d, frame_smooth);
    const int threads = 256;
    const dim3 grid((unsigned)((n + 4 * threads - 1) / (4 * threads)));
    return frames ? xk_launch_pdl(xk_k_noise<true>, grid, dim3(threads), 0, s, cells, col, p)
                  : xk_launch_pdl(xk_k_noise<false>, grid, dim3(threads), 0, s, cells, col, p);
}
