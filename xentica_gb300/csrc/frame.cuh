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

__device__ __forceinline__ bool xk_px_small(int c) { return (uint32_t)c + (1u << 24) < (1u << 25); }

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
// nothing.
__device__ __forceinline__ void xk_store_px4(uint8_t *dst, const uint32_t w[3], int lane, int first, int last)
{
    const uint32_t s = (uint32_t)(uintptr_t)dst & 3u;       // the same in first .. last
    const uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, w[2], 1);
    if (lane < first || lane > last) return;
    uint32_t *a = (uint32_t *)(dst - s);
    if (s == 0) {
        a[0] = w[0];
        a[1] = w[1];
        a[2] = w[2];
        return;
    }
    if (lane > first) {
        a[0] = __funnelshift_l(prev, w[0], 8u * s);
    } else {
        dst[0] = (uint8_t)w[0];
        if (s < 3u) dst[1] = (uint8_t)(w[0] >> 8);
        if (s < 2u) dst[2] = (uint8_t)(w[0] >> 16);
    }
    a[1] = __funnelshift_l(w[0], w[1], 8u * s);
    a[2] = __funnelshift_l(w[1], w[2], 8u * s);
    if (lane == last) {
        dst[11] = (uint8_t)(w[2] >> 24);
        if (s > 1u) dst[10] = (uint8_t)(w[2] >> 16);
        if (s > 2u) dst[9] = (uint8_t)(w[2] >> 8);
    }
}
