// Pieces shared by the kernels that keep colours and write frames
// (MovingAverage, color_effects.py:106-130, and RendererPlain at zoom 1).
#pragma once

#include <stdint.h>

#include "../../include/xk.h"

// max(min(v, old + fade_in), old - fade_out), the sums wrapping
__device__ __forceinline__ int xk_fade(int v, int old, int fade_in, int neg_fade_out)
{
    return __viaddmax_s32(old, neg_fade_out, __viaddmin_s32(old, fade_in, v));
}

// The pixel RendererPlain makes of a colour at zoom 1, in the low byte: the
// colour as a float, / SMOOTH_FACTOR, truncated.  int -> float -> int and a
// division by 1 are exact below 2^24 in magnitude: then it is the colour.
// (Out of line: callers take it only for colours outside xk_px_small.)
static __device__ __noinline__ uint32_t xk_pixel(int c, int smooth)
{
    float f = (float)c;
    if (smooth > 0) f = __fdiv_rn(f, (float)smooth);
    return (uint32_t)(int)f;
}

__host__ __device__ __forceinline__ bool xk_px_small(int c) { return (uint32_t)c + (1u << 24) < (1u << 25); }

// Host: whether every colour that starts below 2^24 in magnitude keeps a
// pixel equal to its low byte (a faded colour lies between the old one and
// the cell's, which is 0 .. 255 smooth here; frames divide by nothing)
inline bool xk_px_stays_small(const xk_desc &d, int frame_smooth)
{
    return frame_smooth <= 1 && d.fade_in >= 0 && d.fade_in <= 1 << 30 && d.fade_out >= 0 &&
           d.fade_out <= 1 << 30 && d.smooth >= 0 && d.smooth < 65536;
}

// Four pixels' low bytes as the three words of their twelve bytes
__device__ __forceinline__ void xk_pack_px4(const uint32_t r[4], const uint32_t g[4], const uint32_t b[4],
                                            uint32_t w[3])
{
    w[0] = __byte_perm(__byte_perm(r[0], g[0], 0x0040), __byte_perm(b[0], r[1], 0x0040), 0x5410);
    w[1] = __byte_perm(__byte_perm(g[1], b[1], 0x0040), __byte_perm(r[2], g[2], 0x0040), 0x5410);
    w[2] = __byte_perm(__byte_perm(b[2], r[3], 0x0040), __byte_perm(g[3], b[3], 0x0040), 0x5410);
}

// Twelve bytes (w[0..2]) of every lane in first .. last to its dst, twelve
// bytes further on from lane to lane, as aligned words wherever the first
// lies: a row of pixels starts at any byte of a frame.  At an offset of s
// bytes from a word each lane writes its bytes after the s that belong to
// its neighbour's last word; the ends go byte by byte.  The whole warp calls
// it (with one row of lanes, or several); lanes outside first .. last store
// nothing.  Streaming stores: frames are read by nobody here (64 noise frames
// of 1920 x 1080 118 -> 105 us).
__device__ __forceinline__ void xk_store_px4(uint8_t *dst, const uint32_t w[3], int lane, int first, int last)
{
    const uint32_t s = (uint32_t)(uintptr_t)dst & 3u;       // the same in first .. last
    const uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, w[2], 1);
    if (lane < first || lane > last) return;
    uint32_t *a = (uint32_t *)(dst - s);
    if (s == 0) {
        __stcs(a + 0, w[0]);
        __stcs(a + 1, w[1]);
        __stcs(a + 2, w[2]);
        return;
    }
    if (lane > first) {
        __stcs(a + 0, __funnelshift_l(prev, w[0], 8u * s));
    } else {
        __stcs(dst + 0, (uint8_t)w[0]);
        if (s < 3u) __stcs(dst + 1, (uint8_t)(w[0] >> 8));
        if (s < 2u) __stcs(dst + 2, (uint8_t)(w[0] >> 16));
    }
    __stcs(a + 1, __funnelshift_l(w[0], w[1], 8u * s));
    __stcs(a + 2, __funnelshift_l(w[1], w[2], 8u * s));
    if (lane == last) {
        __stcs(dst + 11, (uint8_t)(w[2] >> 24));
        if (s > 1u) __stcs(dst + 10, (uint8_t)(w[2] >> 16));
        if (s > 2u) __stcs(dst + 9, (uint8_t)(w[2] >> 8));
    }
}

// The pixels' bytes of the four cells whose colours stand at mine, any
// colours.  (One call out of line: inlined, or called per colour, its
// registers cost the common path 8 %.)
static __device__ __noinline__ uint3 xk_pixels4_any(const int *mine, int smooth)
{
    uint32_t b[3] = {0, 0, 0};
#pragma unroll
    for (int w = 0; w < 3; ++w)
#pragma unroll 1
        for (int k = 0; k < 4; ++k) {
            float f = (float)mine[4 * w + k];
            if (smooth > 0) f = __fdiv_rn(f, (float)smooth);
            b[w] = b[w] >> 8 | (uint32_t)(int)f << 24;
        }
    return make_uint3(b[0], b[1], b[2]);
}

// Whether all twelve are below 2^24 in magnitude
__device__ __forceinline__ bool xk_px_small12(const int c[12])
{
    int lo = min(c[0], c[1]), hi = max(c[0], c[1]);
#pragma unroll
    for (int k = 2; k < 12; k += 2) {
        lo = __vimin3_s32(lo, c[k], c[k + 1]);
        hi = __vimax3_s32(hi, c[k], c[k + 1]);
    }
    return xk_px_small(lo) && xk_px_small(hi);
}

// The pixels' bytes of four cells' colours c, which also stand at mine.
// small: every pixel is its colour's low byte.
__device__ __forceinline__ void xk_pixels4(const int c[12], const int *mine, bool small, int smooth, uint32_t b[3])
{
    uint32_t px[3][4];
#pragma unroll
    for (int k = 0; k < 12; ++k) px[k % 3][k / 3] = (uint32_t)c[k];
    xk_pack_px4(px[0], px[1], px[2], b);
    if (!small) {
        const uint3 v = xk_pixels4_any(mine, smooth);
        b[0] = v.x;
        b[1] = v.y;
        b[2] = v.z;
    }
}

// ---------------------------------------------------------------------------
// A row of colours through shared memory, by a half warp (lane q of 16) whose
// lanes hold four cells each, in lattices whose rows are a multiple of four
// cells: global memory is read and written in the row's 16-byte pieces in order
// (whole sectors a warp; a lane's own 48 bytes at 16 an access touch every
// sector three times), a lane's twelve words are read and written in shared
// memory.

// 16-byte pieces of a buffer for a row of this many cells
__host__ __device__ constexpr int xk_col_pieces(int cells) { return cells / 4 * 3; }

__device__ __forceinline__ void xk_copy_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// Starts the copy of `cells` cells' colours, the first word at col + first
// (cp.async.wait_all ends it)
template <int CELLS>
__device__ __forceinline__ void xk_col_fetch(int4 *buf, const int32_t *col, int64_t first, int cells, int q)
{
    const int4 *at = (const int4 *)(col + first);
#pragma unroll
    for (int k = q; k < xk_col_pieces(CELLS); k += 16)
        if (4 * k < 3 * cells) xk_copy_async16(buf + k, at + k);
}

__device__ __forceinline__ void xk_col_read(const int *mine, int c[12])
{
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int4 o = ((const int4 *)mine)[k];
        c[4 * k] = o.x;
        c[4 * k + 1] = o.y;
        c[4 * k + 2] = o.z;
        c[4 * k + 3] = o.w;
    }
}

__device__ __forceinline__ void xk_col_write(int *mine, const int c[12])
{
#pragma unroll
    for (int k = 0; k < 3; ++k)
        ((int4 *)mine)[k] = make_int4(c[4 * k], c[4 * k + 1], c[4 * k + 2], c[4 * k + 3]);
}

// Stores a row that all its lanes have written (__syncwarp between)
template <int CELLS>
__device__ __forceinline__ void xk_col_store(const int4 *buf, int32_t *col, int64_t first, int cells, int q)
{
    int4 *at = (int4 *)(col + first);
#pragma unroll
    for (int k = q; k < xk_col_pieces(CELLS); k += 16)
        if (4 * k < 3 * cells) at[k] = buf[k];
}
