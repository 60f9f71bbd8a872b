// Pieces shared by the kernels that keep colours and write frames
// (MovingAverage, color_effects.py:106-130, and RendererPlain at zoom 1).
#pragma once

#include <stdint.h>

// max(min(v, old + fade_in), old - fade_out), the sums wrapping
__device__ __forceinline__ int xk_fade(int v, int old, int fade_in, int neg_fade_out)
{
    return __viaddmax_s32(old, neg_fade_out, __viaddmin_s32(old, fade_in, v));
}

// The pixel RendererPlain makes of a colour at zoom 1, in the low byte: the
// colour as a float, / SMOOTH_FACTOR, truncated.  int -> float -> int and a
// division by 1 are exact below 2^24 in magnitude: then it is the colour.
__device__ __forceinline__ uint32_t xk_pixel(int c, int smooth)
{
    if (smooth <= 1 && (uint32_t)c + (1u << 24) < (1u << 25)) return (uint32_t)c;
    float f = (float)c;
    if (smooth > 0) f = __fdiv_rn(f, (float)smooth);
    return (uint32_t)(int)f;
}

// Four pixels' low bytes as the three words of their twelve bytes
__device__ __forceinline__ void xk_pack_px4(const uint32_t r[4], const uint32_t g[4], const uint32_t b[4],
                                            uint32_t w[3])
{
    w[0] = __byte_perm(__byte_perm(r[0], g[0], 0x0040), __byte_perm(b[0], r[1], 0x0040), 0x5410);
    w[1] = __byte_perm(__byte_perm(g[1], b[1], 0x0040), __byte_perm(r[2], g[2], 0x0040), 0x5410);
    w[2] = __byte_perm(__byte_perm(b[2], r[3], 0x0040), __byte_perm(g[3], b[3], 0x0040), 0x5410);
}

// Twelve bytes of every lane (w[0..2]) to dst, lane l's at 12 l from lane 0's,
// as aligned words wherever lane 0's address lies: a frame starts at any byte
// when its pixel count is not a multiple of four.  At an offset of s bytes
// from a word each lane writes its bytes after the s that belong to its
// neighbour's last word; the first and the last lane's ends go byte by byte.
// The whole warp calls it.
__device__ __forceinline__ void xk_store_px4(uint8_t *dst, const uint32_t w[3], int lane)
{
    const uint32_t s = (uint32_t)(uintptr_t)dst & 3u;       // the same in every lane
    uint32_t *a = (uint32_t *)(dst - s);
    if (s == 0) {
        a[0] = w[0];
        a[1] = w[1];
        a[2] = w[2];
        return;
    }
    const uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, w[2], 1);
    if (lane > 0) {
        a[0] = __funnelshift_l(prev, w[0], 8u * s);
    } else {
        dst[0] = (uint8_t)w[0];
        if (s < 3u) dst[1] = (uint8_t)(w[0] >> 8);
        if (s < 2u) dst[2] = (uint8_t)(w[0] >> 16);
    }
    a[1] = __funnelshift_l(w[0], w[1], 8u * s);
    a[2] = __funnelshift_l(w[1], w[2], 8u * s);
    if (lane == 31) {
        dst[11] = (uint8_t)(w[2] >> 24);
        if (s > 1u) dst[10] = (uint8_t)(w[2] >> 16);
        if (s > 2u) dst[9] = (uint8_t)(w[2] >> 8);
    }
}
