// Energy flowing down a gravity field (the reference's GraviCowboys,
// examples/gravicowboys.py:20-71) for sm_103a.
//
// A cell is a uint64 packed LSB first in declaration order
// (properties.py:496-541): energy (12 bits) | new_energy << 12 | gravity
// (float bits) << 24.  One generation, per cell, in the reference's
// arithmetic (its emit and absorb as traced):
//   emit    lowest = 0 + min over the neighbours' gravities (a < b ? a : b, in
//           neighbour order); for buffer k in order, one unit goes to
//           neighbour k when its gravity equals lowest and energy - sent > 0
//           (unsigned); every buffer carries gravity + energy (float);
//           new_energy = energy - sent
//   absorb  energy = (uint16)(new_energy + the units sent towards the cell),
//           gravity = (float)((double)(the float sum of the buffers'
//           gravities in neighbour order) / 8.008)
// and the colour (MovingAverage, color_effects.py:106-130) energy * 255,
// (unsigned)(gravity * 108) twice.  An off-board neighbour of a static border
// reads as the whole border container (border.py:144-151).
//
// One launch per generation.  A block's window is 64 x 32 cells, of which it
// writes the inner 60 x 30: it loads the gravities and energies of the window
// and of a row above and below it into shared memory, runs emit on the window
// (what a cell emits is a byte of units sent, its new energy and the one
// float every buffer carries), then absorb on the inner part.  A thread runs
// four consecutive cells of two rows: rows are read from shared memory 16
// bytes a lane, a quad's edge columns come from the lanes beside it, the
// lowest gravity from column minima shared by neighbouring cells (a window
// that holds a NaN compares in the reference's order instead), the units of
// four cells are gathered bytewise in one word.  Nothing branches on a cell's
// state but a quotient outside the range of the float division.  Colours go
// through shared memory: 48 bytes a lane, but whole sectors a warp both ways,
// and on their way while the states are emitted (16-byte accesses of a lane's
// own 48 bytes ran a generation in 19.0 us, this in 17.2, before the pixels of
// colours beyond 2^24 moved out of line).
//
// 64 frames of 1920 x 1080: 1080 us, against 1410 of one cell a thread (its
// 274 instructions a cell issued at 65 %; now 179, at 56 % of 43 % of the
// warps: what is left to hide is the latency of one short launch a
// generation).  Small lattices, and rows that do not start on 16
// bytes, run one cell a thread (below).
#include "xk_internal.cuh"

#include "frame.cuh"

struct GravParams {
    int32_t W, H;
    int32_t tiles_x;            // tiles a row (a 1-D grid: any height launches)
    uint64_t border;            // off-board container (static border)
    int32_t color_kind;         // XK_COLOR_*
    int32_t fade_in, neg_fade_out, smooth;
    uint32_t red;               // 255 smooth
    uint8_t *frame;             // null, or the W x H RendererPlain frame (zoom 1, no offset)
    int32_t frame_smooth;       // its SMOOTH_FACTOR (0: none)
};

#define XK_GC_WX 64             // window
#define XK_GC_WY 32
#define XK_GC_IX 60             // its inner part: columns 2 .. 61, rows 1 .. 30
#define XK_GC_IY 30
#define XK_GC_THREADS 256
#define XK_GC_GP 64             // row pitches: gravities,
#define XK_GC_P 72              // entries, and bytes of the units sent
#define XK_GC_PB 96

// neighbours in the reference's order (x, y): (-1,-1) (-1,0) (-1,1) (0,-1)
// (0,1) (1,-1) (1,0) (1,1); neighbour 7 - k points back along k

__device__ __forceinline__ float xk_gc_grav(uint64_t c) { return __uint_as_float((uint32_t)(c >> 24)); }

// (float)((double)f / 8.008) in float arithmetic (the double-precision pipe
// is narrow on this part), for |f| in [2^-60, 2^120]: the quotient as the
// unevaluated sum q1 + t (8.008 split as CH + CL, R = RN(1/8.008); the
// remainder f - q1 * 8.008 by two fmas), relative error below 2^-45.  When
// q1 + t less and plus 2^-43 q1 round to the same float, the exact quotient,
// and its double rounding, lie between them and round to it (rounding is
// monotone; the two sums' own terms are rounded by less than 2^-46 q1).
// False, as for an infinity or a NaN: the division itself has to be taken.
// Checked equal to the double division for every float of that range (it
// declines none).
__device__ __forceinline__ bool xk_gc_mean(float f, float &s)
{
    constexpr float CH = 0x1.00418ap+3f, CL = -0x1.916872p-22f, R = 0x1.ff7d1p-4f;
    const float q1 = __fmul_rn(f, R);
    const float e = __fmaf_rn(-q1, CH, f);
    const float e2 = __fmaf_rn(-q1, CL, e);
    const float t = __fmul_rn(e2, R);
    s = __fadd_rn(q1, __fmaf_rn(q1, 0x1p-43f, t));
    return s == __fadd_rn(q1, __fmaf_rn(q1, -0x1p-43f, t));
}

__device__ __noinline__ float xk_gc_mean_f64(float f) { return __double2float_rn(__ddiv_rn((double)f, 8.008)); }

// 1 where the two are equal (no NaN), else 0, in one instruction
__device__ __forceinline__ float xk_gc_equal(float a, float b)
{
    float r;
    asm("set.eq.f32.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

struct __align__(16) GravTile {
    float g[XK_GC_WY + 2][XK_GC_GP];            // gravities: window row r at r + 1
    uint16_t e[XK_GC_WY + 2][XK_GC_P];          // energies, then new energies; column c at c + 2
    float y[XK_GC_WY][XK_GC_P];                 // the gravity every buffer carries; column c at c + 2
    uint8_t sent[XK_GC_WY][XK_GC_PB];           // units sent, by neighbour as xk_gc_bit; column c at c + 2
    int4 col[XK_GC_IY][xk_col_pieces(XK_GC_IX)];    // colours of the inner part (frame.cuh)
};

// The bit of a sent byte that stands for a unit to neighbour j
__host__ __device__ constexpr uint32_t xk_gc_bit(int j)
{
    return j == 0 ? 8u : j == 1 ? 128u : j == 2 ? 2u : j == 3 ? 32u : j == 4 ? 4u : j == 5 ? 64u : j == 6 ? 1u : 16u;
}

// What a cell with this energy sends to its ties (neighbours of the lowest
// gravity; nibble j's top bit: neighbour j), as a sent byte in the low byte:
// one unit each, in neighbour order, while energy lasts.  A nibble of
// ties * 0x02222222 counts the ties before it (0 .. 7); energy (up to 8) + 7
// less the count keeps its top bit exactly when the count is below energy.
__device__ __forceinline__ uint32_t xk_gc_sent(uint32_t energy, uint32_t ties)
{
    const uint32_t m = (min(energy, 8u) * 0x11111111u + 0x77777777u - ties * 0x02222222u) & ties;
    const uint32_t t = m | m >> 17;
    return (t | t >> 10) & 0xFFu;
}

// The lowest of a cell's neighbours' gravities by the reference's comparisons
// (at: the one above and to the left in the loaded tile)
static __device__ __noinline__ float xk_gc_lowest(const float *at)
{
    float m = *at;
#pragma unroll 1
    for (int j = 1; j < 8; ++j) {
        const int c = j + (j > 3);          // of the 3 x 3, column by column
        const float n = at[c % 3 * XK_GC_GP + c / 3];
        m = m < n ? m : n;
    }
    return m;
}

template <bool TORUS>
__global__ void __launch_bounds__(XK_GC_THREADS, 3)
xk_k_gravity(const uint64_t *__restrict__ src, uint64_t *__restrict__ dst, int32_t *__restrict__ col,
             GravParams p)
{
    __shared__ GravTile T;
    constexpr int WARPS = XK_GC_THREADS / 32, HALVES = XK_GC_THREADS / 16;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int by = blockIdx.x / p.tiles_x, bx = blockIdx.x - by * p.tiles_x;
    const int x0 = bx * XK_GC_IX - 2, y0 = by * XK_GC_IY - 1;     // the window's first cell
    const int q = lane & 15, half = tid >> 4;       // quad of a row, half warp

    // a warp a row, two cells a lane (one access where rows start on 16 bytes)
    constexpr int ROWS = (XK_GC_WY + 2 + WARPS - 1) / WARPS;
    int gx[2];
    bool xin[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        gx[k] = x0 + 2 * lane + k;
        xin[k] = (unsigned)gx[k] < (unsigned)p.W;
        if (!xin[k]) {
            if (TORUS) {
                gx[k] %= p.W;
                if (gx[k] < 0) gx[k] += p.W;
            } else {
                gx[k] = 0;
            }
        }
    }
    xk_grid_dep_wait();                 // launched as a dependent of the previous generation
    const bool colours = p.color_kind != XK_COLOR_NONE;
    const int width = min(XK_GC_IX, p.W - (x0 + 2));        // cells of a row of the inner part
    if (colours)
#pragma unroll
        for (int r = half; r < XK_GC_IY; r += HALVES) {
            const int gy = y0 + 1 + r;
            if (gy < p.H)
                xk_col_fetch<XK_GC_IX>(T.col[r], col, 3 * ((int64_t)gy * p.W + x0 + 2), width, q);
        }
    uint64_t v[ROWS][2];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const int r = wid + i * WARPS;
        int gy = y0 + r - 1;
        const bool yin = (unsigned)gy < (unsigned)p.H;
        if (!yin) {
            if (TORUS) {
                gy %= p.H;
                if (gy < 0) gy += p.H;
            } else {
                gy = 0;
            }
        }
        const uint64_t *row = src + (int64_t)gy * p.W;
        if (r < XK_GC_WY + 2) {
            const ulonglong2 w = __ldg((const ulonglong2 *)(row + gx[0]));
            v[i][0] = w.x;
            v[i][1] = w.y;
        }
        if (!TORUS) {
            if (!(xin[0] && yin)) v[i][0] = p.border;
            if (!(xin[1] && yin)) v[i][1] = p.border;
        }
    }
    bool nan = false;
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const int r = wid + i * WARPS;
        if (r < XK_GC_WY + 2) {
            const float a = xk_gc_grav(v[i][0]), b = xk_gc_grav(v[i][1]);
            nan |= a != a || b != b;
            *(float2 *)&T.g[r][2 * lane] = make_float2(a, b);
            *(uint32_t *)&T.e[r][2 * lane + 2] =
                __byte_perm((uint32_t)v[i][0], (uint32_t)v[i][1], 0x5410) & 0x0FFF0FFFu;
        }
    }
    const bool ordered = __syncthreads_or(nan);

    // emit.  The window's first and last columns take a neighbour from the
    // other row of lanes; absorb reads what columns 1 .. 62 emit.
#pragma unroll
    for (int er = half; er < XK_GC_WY; er += HALVES) {
        float f[3][6];      // rows er - 1 .., columns 4 q - 1 .. 4 q + 4
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float4 m = *(const float4 *)&T.g[er + a][4 * q];
            f[a][0] = __shfl_up_sync(0xFFFFFFFFu, m.w, 1);
            f[a][1] = m.x;
            f[a][2] = m.y;
            f[a][3] = m.z;
            f[a][4] = m.w;
            f[a][5] = __shfl_down_sync(0xFFFFFFFFu, m.x, 1);
        }
        float ud[6], all[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            ud[c] = fminf(f[0][c], f[2][c]);
            all[c] = fminf(ud[c], f[1][c]);
        }
        const uint32_t ew[2] = {*(const uint32_t *)&T.e[er + 1][4 * q + 2],
                                *(const uint32_t *)&T.e[er + 1][4 * q + 4]};
        uint32_t sent[4], newe[4];
        float y[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float n[8] = {f[0][k], f[1][k], f[2][k], f[0][k + 1], f[2][k + 1],
                                f[0][k + 2], f[1][k + 2], f[2][k + 2]};
            float m = fminf(fminf(all[k], ud[k + 1]), all[k + 2]);
            if (ordered) m = xk_gc_lowest(&T.g[er][max(4 * q + k - 1, 0)]);
            const float lowest = __fadd_rn(0.0f, m);
            // ties summed as bits of two floats' mantissas, on the fma pipe
            float lo = 8388608.0f, hi = 8388608.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                lo = __fmaf_rn(xk_gc_equal(lowest, n[j]), (float)(8 << (4 * j)), lo);
                hi = __fmaf_rn(xk_gc_equal(lowest, n[j + 4]), (float)(8 << (4 * j)), hi);
            }
            const uint32_t ties = __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x5410);
            const uint32_t energy = (k & 1) ? ew[k >> 1] >> 16 : ew[k >> 1] & 0xFFFFu;
            sent[k] = xk_gc_sent(energy, ties);
            newe[k] = energy - (uint32_t)__popc(sent[k]);
            y[k] = __fadd_rn(f[1][k + 1], (float)energy);
        }
        if (!TORUS) {
            // off-board neighbours read as the border container: its
            // gravity is carried, its energy sent (added in absorb)
            const int gy = y0 + er;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if ((unsigned)gy >= (unsigned)p.H || (unsigned)(x0 + 4 * q + k) >= (unsigned)p.W) {
                    sent[k] = 0;
                    y[k] = __uint_as_float((uint32_t)(p.border >> 24));
                }
        }
        *(uint32_t *)&T.e[er + 1][4 * q + 2] = newe[0] | newe[1] << 16;
        *(uint32_t *)&T.e[er + 1][4 * q + 4] = newe[2] | newe[3] << 16;
        *(float2 *)&T.y[er][4 * q + 2] = make_float2(y[0], y[1]);
        *(float2 *)&T.y[er][4 * q + 4] = make_float2(y[2], y[3]);
        *(uint16_t *)&T.sent[er][4 * q + 2] = (uint16_t)(sent[0] | sent[1] << 8);
        *(uint16_t *)&T.sent[er][4 * q + 4] = (uint16_t)(sent[2] | sent[3] << 8);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    // absorb: row r + 1 of the window, columns 4 q + 2 ..; a half warp's last
    // quad, and rows past the inner part, run on what is there and store
    // nothing (whole warps exchange columns and pixels)
    const int ox = x0 + 2 + 4 * q;
#pragma unroll
    for (int r = half; r < XK_GC_WY; r += HALVES) {
        const int gy = y0 + 1 + r, top = min(r, XK_GC_IY - 1);
        const bool row_in = r < XK_GC_IY && gy < p.H, in = row_in && q < 15 && ox < p.W;
        float y[3][6];                      // columns 4 q + 1 .. 4 q + 6
        uint32_t sl[3], sc[3], sr[3];       // sent bytes of columns one less, equal, one more
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float *at = &T.y[top + a][4 * q + 4];
            const float4 m = *(const float4 *)at;
            y[a][0] = __shfl_up_sync(0xFFFFFFFFu, m.w, 1);
            if (q == 0) y[a][0] = at[-1];
            y[a][1] = m.x;
            y[a][2] = m.y;
            y[a][3] = m.z;
            y[a][4] = m.w;
            y[a][5] = __shfl_down_sync(0xFFFFFFFFu, m.x, 1);
            const uint32_t *s = (const uint32_t *)&T.sent[top + a][4 * q];
            sc[a] = s[1];
            sl[a] = __byte_perm(s[0], s[1], 0x6543);
            sr[a] = __byte_perm(s[1], s[2], 0x4321);
        }
        // neighbour j's unit towards a cell is its unit to its neighbour 7 - j
        constexpr uint32_t EACH = 0x01010101u;
        const uint32_t got = (sl[0] & EACH * xk_gc_bit(7)) | (sl[1] & EACH * xk_gc_bit(6)) |
                             (sl[2] & EACH * xk_gc_bit(5)) | (sc[0] & EACH * xk_gc_bit(4)) |
                             (sc[2] & EACH * xk_gc_bit(3)) | (sr[0] & EACH * xk_gc_bit(2)) |
                             (sr[1] & EACH * xk_gc_bit(1)) | (sr[2] & EACH * xk_gc_bit(0));
        const uint2 ne = *(const uint2 *)&T.e[top + 2][4 * q + 4];
        float field[4], g[4];
        bool sure = true;
        float least = 0x1p-60f, most = 0x1p+120f;       // of the fields' magnitudes
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float n[8] = {y[0][k], y[1][k], y[2][k], y[0][k + 1], y[2][k + 1],
                                y[0][k + 2], y[1][k + 2], y[2][k + 2]};
            field[k] = 0.0f;
#pragma unroll
            for (int j = 0; j < 8; ++j) field[k] = __fadd_rn(field[k], n[j]);
            sure &= xk_gc_mean(field[k], g[k]);
            least = fminf(least, fabsf(field[k]));
            most = fmaxf(most, fabsf(field[k]));
        }
        // (a sum of buffers starts from +0: it is never -0, whose quotient
        // the float arithmetic would make +0)
        if ((!sure || least < 0x1p-60f || most > 0x1p+120f) && in)
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (field[k] != 0.0f) g[k] = xk_gc_mean_f64(field[k]);
        const int64_t i = (int64_t)gy * p.W + ox;
        uint64_t out[4];
        uint32_t energy[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            uint32_t received = (uint32_t)__popc(got & (0xFFu << (8 * k)));
            if (!TORUS) {
                const int cols = 1 + (ox + k > 0) + (ox + k + 1 < p.W), rows = 1 + (gy > 0) + (gy + 1 < p.H);
                received += (uint32_t)(9 - cols * rows) * ((uint32_t)p.border & 4095u);
            }
            const uint32_t nw = k < 2 ? ne.x : ne.y;
            const uint32_t newe = (k & 1) ? nw >> 16 : nw & 0xFFFFu;
            energy[k] = TORUS ? newe + received : (newe + received) & 0xFFFFu;
            out[k] = (uint64_t)(energy[k] & 4095u) | (uint64_t)newe << 12 | (uint64_t)__float_as_uint(g[k]) << 24;
        }
        if (in)
            asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(dst + i), "l"(out[0]), "l"(out[1]),
                         "l"(out[2]), "l"(out[3])
                         : "memory");
        if (!colours) continue;
        const int64_t first = 3 * ((int64_t)gy * p.W + x0 + 2);
        int *mine = (int *)T.col[top] + 12 * min(q, 14);
        int c[12];
        xk_col_read(mine, c);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int gg = (int)__float2uint_rz(__fmul_rn(g[k], 108.0f)) * p.smooth;
            c[3 * k] = xk_fade((int)(energy[k] * p.red), c[3 * k], p.fade_in, p.neg_fade_out);
            c[3 * k + 1] = xk_fade(gg, c[3 * k + 1], p.fade_in, p.neg_fade_out);
            c[3 * k + 2] = xk_fade(gg, c[3 * k + 2], p.fade_in, p.neg_fade_out);
        }
        if (in) xk_col_write(mine, c);
        __syncwarp();
        if (row_in) xk_col_store<XK_GC_IX>(T.col[r], col, first, width, q);
        if (!p.frame) continue;
        uint32_t b[3];
        xk_pixels4(c, mine, p.frame_smooth <= 1 && xk_px_small12(c), p.frame_smooth, b);
        const int left = lane & 16;                     // the row's half warp
        uint8_t *at = p.frame + 3 * i;
        xk_store_px4(at, b, lane, left, row_in ? left + width / 4 - 1 : -1);
    }
}

// ---------------------------------------------------------------------------
// One cell a thread on 32 x 32 tiles with a halo of two: lattices of too few
// windows to fill the chip, and rows that do not start on 16 bytes
// (xk_gravity_step's rule).

// the Moore deltas in the reference's order (x, y): (-1,-1) (-1,0) (-1,1)
// (0,-1) (0,1) (1,-1) (1,0) (1,1); neighbour 7 - k points back along k
__device__ __forceinline__ int xk_gc_dx(int k) { return k < 3 ? -1 : k < 5 ? 0 : 1; }
__device__ __forceinline__ int xk_gc_dy(int k) { return (k == 0 || k == 3 || k == 5) ? -1 : (k == 1 || k == 6) ? 0 : 1; }

// the quotient of any field (zeros keep their sign)
__device__ __forceinline__ float xk_gc_mean_any(float f)
{
    float s;
    if (xk_gc_mean(f, s) && fabsf(f) >= 0x1p-60f && fabsf(f) <= 0x1p+120f) return s;
    return f == 0.0f ? f : xk_gc_mean_f64(f);
}

#define XK_GC1_TX 32
#define XK_GC1_TY 32            // rows of a tile; each of the 8 warps runs four of them

struct GravTileOne {
    float g[XK_GC1_TY + 4][XK_GC1_TX + 4];        // gravities, halo of two
    uint32_t e[XK_GC1_TY + 4][XK_GC1_TX + 4];     // energies
    // emitted: .x units sent (bit k: to neighbour k) | new_energy << 8, .y the
    // bits of the gravity every buffer carries (one 64-bit load in absorb)
    uint2 x[XK_GC1_TY + 2][XK_GC1_TX + 2];
};

// emit of the cell at tile position (y, x): the units go to the neighbours of
// the lowest gravity in neighbour order, one each while energy lasts, i.e. to
// the first min(energy, ties) of them
__device__ __forceinline__ void xk_gc_emit(GravTileOne &T, int y, int x, int ey, int ex)
{
    const uint32_t energy = T.e[y][x];
    float gk[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) gk[k] = T.g[y + xk_gc_dy(k)][x + xk_gc_dx(k)];
    float m = gk[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) m = m < gk[k] ? m : gk[k];
    const float lowest = __fadd_rn(0.0f, m);
    uint32_t ties = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) ties |= (uint32_t)(lowest == gk[k]) << k;
    uint32_t mask = ties;
    if (energy < (uint32_t)__popc(ties)) {       // energy < 8: only its first set bits
        uint32_t rest = ties;
        mask = 0;
        for (uint32_t j = 0; j < energy; ++j) {
            const uint32_t low = rest & (0u - rest);
            mask |= low;
            rest ^= low;
        }
    }
    T.x[ey][ex] = make_uint2(mask | (energy - (uint32_t)__popc(mask)) << 8,
                             __float_as_uint(__fadd_rn(T.g[y][x], (float)energy)));
}

template <bool TORUS>
__global__ void __launch_bounds__(XK_GC_THREADS)
xk_k_gravity_one(const uint64_t *__restrict__ src, uint64_t *__restrict__ dst, int32_t *__restrict__ col,
             GravParams p)
{
    __shared__ GravTileOne T;
    const int tid = threadIdx.y * XK_GC1_TX + threadIdx.x;
    const int x0 = blockIdx.x * XK_GC1_TX, y0 = blockIdx.y * XK_GC1_TY;
    xk_grid_dep_wait();                 // launched as a dependent of the previous generation
    for (int e = tid; e < (XK_GC1_TY + 4) * (XK_GC1_TX + 4); e += XK_GC_THREADS) {
        const int sy = e / (XK_GC1_TX + 4), sx = e % (XK_GC1_TX + 4);
        int gx = x0 + sx - 2, gy = y0 + sy - 2;
        uint64_t v;
        if (TORUS) {
            if ((unsigned)gx >= (unsigned)p.W) { gx %= p.W; if (gx < 0) gx += p.W; }
            if ((unsigned)gy >= (unsigned)p.H) { gy %= p.H; if (gy < 0) gy += p.H; }
            v = __ldg(src + (int64_t)gy * p.W + gx);
        } else {
            v = (gx >= 0 && gx < p.W && gy >= 0 && gy < p.H) ? __ldg(src + (int64_t)gy * p.W + gx) : p.border;
        }
        T.g[sy][sx] = xk_gc_grav(v);
        T.e[sy][sx] = (uint32_t)v & 4095u;
    }
    __syncthreads();
    for (int e = tid; e < (XK_GC1_TY + 2) * (XK_GC1_TX + 2); e += XK_GC_THREADS) {
        const int ey = e / (XK_GC1_TX + 2), ex = e % (XK_GC1_TX + 2);
        xk_gc_emit(T, ey + 1, ex + 1, ey, ex);   // off-board positions are never read
    }
    __syncthreads();
    const int gx = x0 + threadIdx.x;
    if (gx >= p.W) return;
#pragma unroll
    for (int r = 0; r < XK_GC1_TY / 8; ++r) {
        const int ly = threadIdx.y + 8 * r, gy = y0 + ly;
        if (gy >= p.H) return;
        const int ty = ly + 1, tx = threadIdx.x + 1;
        uint32_t got = 0, received = 0;
        float gk[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int dx = xk_gc_dx(k), dy = xk_gc_dy(k);
            const bool on = TORUS || ((unsigned)(gx + dx) < (unsigned)p.W && (unsigned)(gy + dy) < (unsigned)p.H);
            if (on) {
                const uint2 w = T.x[ty + dy][tx + dx];
                got |= w.x & (1u << (7 - k));   // the unit neighbour k sent back along k
                gk[k] = __uint_as_float(w.y);
            } else {
                received += (uint32_t)p.border & 4095u;
                gk[k] = xk_gc_grav(p.border);
            }
        }
        received += (uint32_t)__popc(got);
        float field = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) field = __fadd_rn(field, gk[k]);
        const uint32_t newe = T.x[ty][tx].x >> 8;
        const uint32_t energy = (newe + received) & 0xFFFFu;
        const float g = xk_gc_mean_any(field);
        const int64_t i = (int64_t)gy * p.W + gx;
        dst[i] = (uint64_t)(energy & 4095u) | (uint64_t)newe << 12 | (uint64_t)__float_as_uint(g) << 24;
        if (p.color_kind == XK_COLOR_NONE) continue;
        const int gg = (int)__float2uint_rz(__fmul_rn(g, 108.0f));
        int rgb[3] = {(int)energy * 255 * p.smooth, gg * p.smooth, gg * p.smooth};
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            const int old = col[3 * i + ch];
            const int m = rgb[ch] < old + p.fade_in ? rgb[ch] : old + p.fade_in;
            rgb[ch] = m > old - (int)(0u - (uint32_t)p.neg_fade_out) ? m : old - (int)(0u - (uint32_t)p.neg_fade_out);
        }
        col[3 * i] = rgb[0];
        col[3 * i + 1] = rgb[1];
        col[3 * i + 2] = rgb[2];
        if (p.frame) {
            // RendererPlain at zoom 1: the colour as a float, / SMOOTH_FACTOR,
            // truncated, its low byte; exact without the division below 2^24
            const bool small = (((uint32_t)rgb[0] + (1u << 24)) | ((uint32_t)rgb[1] + (1u << 24)) |
                                ((uint32_t)rgb[2] + (1u << 24))) < (1u << 25);
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                uint8_t px;
                if (p.frame_smooth <= 1 && small) {
                    px = (uint8_t)rgb[ch];
                } else {
                    float v = (float)rgb[ch];
                    if (p.frame_smooth > 0) v = __fdiv_rn(v, (float)p.frame_smooth);
                    px = (uint8_t)(int)v;
                }
                p.frame[3 * i + ch] = px;
            }
        }
    }
}

cudaError_t xk_gravity_step(const uint64_t *src, uint64_t *dst, int32_t *col, const xk_desc &d,
                            cudaStream_t s, uint8_t *frame, int frame_smooth)
{
    GravParams p;
    p.W = (int32_t)d.size[0];
    p.H = (int32_t)d.size[1];
    p.border = d.border_value;
    p.color_kind = d.color_kind;
    p.fade_in = d.fade_in;
    p.neg_fade_out = (int32_t)(0u - (uint32_t)d.fade_out);
    p.smooth = d.smooth;
    p.red = 255u * (uint32_t)d.smooth;
    p.frame = frame;
    p.frame_smooth = frame_smooth;
    // Four cells a thread where rows start on 16 bytes and the windows are two
    // or more an SM: with fewer a generation takes 4.6 to 8.3 us by where the
    // blocks land (640 x 360, 60 generations: 278 to 424 us, 333 x 222 500, against 412 and
    // 400 one cell a thread), and colours by words gain nothing (1325 x 500
    // 634 to 643 against 623 to 631).  1324 x 500 545 against 635, 1920 x 1080
    // 1 010 against 1 300.
    const int64_t tiles_x = ((int64_t)p.W + XK_GC_IX - 1) / XK_GC_IX;
    const int64_t tiles = tiles_x * (((int64_t)p.H + XK_GC_IY - 1) / XK_GC_IY);
    p.tiles_x = (int32_t)tiles_x;
    if (p.W % 4 != 0 || !xk_tiles_in_range(p.W, p.H) || tiles < 2 * (int64_t)xk_sm_count()) {
        const dim3 one(XK_GC1_TX, XK_GC_THREADS / XK_GC1_TX);
        const dim3 over((p.W + XK_GC1_TX - 1) / XK_GC1_TX, (p.H + XK_GC1_TY - 1) / XK_GC1_TY);
        return d.torus ? xk_launch_pdl(xk_k_gravity_one<true>, over, one, 0, s, src, dst, col, p)
                       : xk_launch_pdl(xk_k_gravity_one<false>, over, one, 0, s, src, dst, col, p);
    }
    const dim3 block(XK_GC_THREADS), grid((unsigned)tiles);
    return d.torus ? xk_launch_pdl(xk_k_gravity<true>, grid, block, 0, s, src, dst, col, p)
                   : xk_launch_pdl(xk_k_gravity<false>, grid, block, 0, s, src, dst, col, p);
}
