// EvoLife generation kernel for sm_103a.
//
// Restates, per cell and in the same operation order, the absorb + colour
// program the reference generates for EvoLife (examples/evolife.py:20-128,
// tools/genetics.py:7-56, tools/color.py:8-125):
//   cell = energy (9 bits) | rule (18 bits) << 9 | rng (16 bits) << 27, uint64
//   (properties.py:496-541); 2-D Moore torus, neighbour k at the reference's
//   delta order (-1,-1) (-1,0) (-1,1) (0,-1) (0,1) (1,-1) (1,0) (1,1).
// Emit copies energy and rule to every buffer, so a neighbour's buffer is its
// main state: emit is fused away and the kernel reads neighbours directly
// (ping-pong state buffers).  Every read of the cell's RandomProperty advances
// x = (x * 58321 + 11113) % 65535 (properties.py:638-660): once for the start
// gene, then once per gene (twice with mutation).  Floats follow IEEE
// round-to-nearest with no contraction (__fdiv_rn, __fmul_rn, __fadd_rn).
//
// The crossover's draws depend only on the cell's 16-bit random state x0 at
// the start of the crossover and on the number n of parents: the start gene,
// and for every gene which parent wins it (and, with mutation, whether it
// mutates).  So for every (x0, n) they are precomputed once per process, on
// the device: the winner of each gene as three bit planes and the start gene
// in one 64-bit word, 4.2 MB that stay in L2.  A cell's crossover is then a
// tree of bitwise selects over its parents -- the genes in visiting order,
// before the max_genes cut -- followed by keeping the first max_genes set
// genes in visiting order and the mutation flips.  The state after the
// crossover is one composed affine map of x0.
//
// On large lattices a thread runs four consecutive cells of a row, so that
// what is a byte per neighbour is computed for four cells in one word: the
// counts of living neighbours, and the bit-sliced counts of the eight birth
// bits (one carry-save tree).  A block's 64 x 16 cells and their halo lie in shared memory: a
// cell's parents are read from there in slot order, at offsets that a table
// gives by the mask of its parents.  Colours go through shared memory in
// whole sectors (frame.cuh).
//
// 64 frames of 1920 x 1080: 1444 us with four cells a thread, 1630 with one,
// against 1961 when a parent's won genes were a mask of their own, loaded for
// each (429 instructions a cell, issued at 71 %; now 270, at 54 %: the random
// reads of the crossover's table, one sector a cell with a parent, and the
// two shared-memory passes are what it waits for).  256 x 256: 237 -> 190.
#include <string.h>

#include <map>
#include <mutex>
#include <utility>

#include "xk_internal.cuh"

#include "frame.cuh"

// GenomeColor.positional weights (double) per gene and channel
__constant__ double c_evo_pos[18 * 3];

__device__ __forceinline__ uint32_t xk_lcg(uint32_t x) { return (x * 58321u + 11113u) % 65535u; }

// float -> unsigned int as the GPU converts: truncation, NaN -> 0
__device__ __forceinline__ uint32_t xk_f2u(float v) { return __float2uint_rz(v); }

// bit j of the result = bit (s + j) mod 18 of v (v < 2^18, s < 18), and back
__device__ __forceinline__ uint32_t xk_rot18(uint32_t v, uint32_t s)
{
    return ((v >> s) | (v << (18u - s))) & 0x3FFFFu;
}

__device__ __forceinline__ uint32_t xk_unrot18(uint32_t w, uint32_t s)
{
    return ((w << s) | (w >> (18u - s))) & 0x3FFFFu;
}

// hsv2rgb(hue, 1, 1) with deferred hue (tools/color.py:8-60) of the modular
// genome colour's hue (rule >> 1) % 360: the float channels before EvoLife's
// energy weighting
__device__ __forceinline__ void xk_evo_hue_rgb(uint32_t hue, float *out)
{
    float hue_f = 0.0f;
    hue_f = __fadd_rn(hue_f, __fmul_rn(__fdiv_rn((float)hue, 360.0f), 6.0f));
    uint32_t hue_i = 0;
    hue_i += xk_f2u(hue_f);
    hue_f = __fsub_rn(hue_f, (float)hue_i);
    float sat = 0.0f;
    sat = __fadd_rn(sat, 1.0f);
    float val = 0.0f;
    val = __fadd_rn(val, 1.0f);
    float grad_p = 0.0f, grad_q = 0.0f, grad_t = 0.0f;
    grad_p = __fadd_rn(grad_p, __fmul_rn(val, __fsub_rn(1.0f, sat)));
    grad_q = __fadd_rn(grad_q, __fmul_rn(val, __fsub_rn(1.0f, __fmul_rn(sat, hue_f))));
    grad_t = __fadd_rn(grad_t, __fmul_rn(val, __fsub_rn(1.0f, __fmul_rn(sat, __fsub_rn(1.0f, hue_f)))));
    float r = __fmul_rn((float)((hue_i == 0) | (hue_i >= 5)), val);
    r = __fadd_rn(r, __fmul_rn((float)(hue_i == 1), grad_q));
    r = __fadd_rn(r, __fmul_rn((float)((hue_i == 2) | (hue_i == 3)), grad_p));
    r = __fadd_rn(r, __fmul_rn((float)(hue_i == 4), grad_t));
    float g = __fmul_rn((float)((hue_i == 0) | (hue_i >= 6)), grad_t);
    g = __fadd_rn(g, __fmul_rn((float)((hue_i == 1) | (hue_i == 2)), val));
    g = __fadd_rn(g, __fmul_rn((float)(hue_i == 3), grad_q));
    g = __fadd_rn(g, __fmul_rn((float)((hue_i == 4) | (hue_i == 5)), grad_p));
    float b = __fmul_rn((float)(((hue_i == 0) | (hue_i == 1)) | (hue_i >= 6)), grad_p);
    b = __fadd_rn(b, __fmul_rn((float)(hue_i == 2), grad_t));
    b = __fadd_rn(b, __fmul_rn((float)((hue_i == 3) | (hue_i == 4)), val));
    b = __fadd_rn(b, __fmul_rn((float)(hue_i == 5), grad_q));
    out[0] = r;
    out[1] = g;
    out[2] = b;
}

// the 360 hues' channels, computed once per device context by the same
// operations (xk_k_evo_hues) and read per cell
__global__ void xk_k_evo_hues(float4 *__restrict__ hues)
{
    const uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= 360u) return;
    float c[3];
    xk_evo_hue_rgb(h, c);
    hues[h] = make_float4(c[0], c[1], c[2], 0.0f);
}

// modular genome colour with the energy weighting of EvoLife.color
// (evolife.py:431-444)
__device__ __forceinline__ int3 xk_evo_color_modular(const float4 *hues, uint32_t rule,
                                                     uint32_t energy)
{
    const bool shown = rule != 0 && energy < 255u;
    float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (shown) c = hues[(rule >> 1) % 360u];
    const float e = (float)(255 - (int)energy);
    return make_int3((int)xk_f2u(__fmul_rn(c.x, e)), (int)xk_f2u(__fmul_rn(c.y, e)), (int)xk_f2u(__fmul_rn(c.z, e)));
}

// GenomeColor.positional (tools/color.py:63-104): double weights added into
// float variables, then normalised by the float maximum
static __device__ __noinline__ int3 xk_evo_color_positional(uint32_t rule, uint32_t energy)
{
    float red = 0.0f, green = 0.0f, blue = 0.0f;
#pragma unroll
    for (int i = 0; i < 18; ++i) {
        if ((rule >> i) & 1u) {
            red = __double2float_rn(__dadd_rn((double)red, c_evo_pos[3 * i]));
            green = __double2float_rn(__dadd_rn((double)green, c_evo_pos[3 * i + 1]));
            blue = __double2float_rn(__dadd_rn((double)blue, c_evo_pos[3 * i + 2]));
        }
    }
    float maxval = 0.0f;
    const float m01 = red > green ? red : green;
    maxval = __fadd_rn(maxval, m01 > blue ? m01 : blue);
    red = __fdiv_rn(red, maxval);
    green = __fdiv_rn(green, maxval);
    blue = __fdiv_rn(blue, maxval);
    const int e = (255 - (int)energy) * ((int)(rule > 0) * (int)(energy < 255));
    return make_int3((int)xk_f2u(__fmul_rn(red, (float)e)), (int)xk_f2u(__fmul_rn(green, (float)e)),
                     (int)xk_f2u(__fmul_rn(blue, (float)e)));
}

// The random draws of the crossover are u(x) = RN(x / 65535) of the 16-bit
// state x in [0, 65534]: a parent index trunc(RN(u(x) * n)) for n parents,
// the start gene trunc(RN(u(x) * 18)) % 8, and a mutation iff u(x) <= t.
// For each n (and 18) there is a multiplier K with floor(x * K / 2^32) equal
// to the float expression for every x -- found once per process on the host
// by trying multipliers near n * 2^32 / 65535 against all 65535 states with
// the same IEEE single-precision operations -- so a draw is one umulhi.  The
// mutation test is monotonic in x: x <= mut_x.
struct EvoParams {
    int32_t W, H;
    int32_t tiles_x;           // tiles a row (a 1-D grid: any height launches)
    uint32_t death_speed, max_genes;
    int32_t mut_x;             // largest x with u(x) <= t (-1: none)
    int32_t mutation;          // mutation_prob > 0
    int32_t positional;
    int32_t color_kind;        // XK_COLOR_*
    int32_t fade_in, neg_fade_out, smooth;
    uint32_t kmul[9];          // parent draw for 0..8 parents (0: none)
    uint32_t kstart;           // start-gene draw (n = 18)
    uint32_t jump_a, jump_c;   // the crossover's RNG advances as one map x -> (a x + c) % 65535
    const uint2 *won;          // winners' bit planes and start gene per x0, blocks of 65536 x0 per n
    const uint4 *slots;        // parents' offsets in shared memory per mask of parents
    const uint32_t *mut;       // mutation flips per x0 (mutation only)
    const float4 *hues;        // modular colour channels per hue
    uint8_t *frame;            // null, or the W x H RendererPlain frame (zoom 1, no offset)
    int32_t frame_smooth;      // its SMOOTH_FACTOR (0: none)
    int32_t small;             // every colour is below 2^24 in magnitude and its pixel's value
};

static float evo_u(uint32_t x) { return (float)x / 65535.0f; }

// K with floor(x * K / 2^32) == trunc(RN(u(x) * n)) for all x in [0, 65534]
static uint32_t evo_find_multiplier(uint32_t n)
{
    static uint32_t want[65535];
    for (uint32_t x = 0; x < 65535; ++x) want[x] = (uint32_t)(evo_u(x) * (float)n);
    const uint64_t base = ((uint64_t)n << 32) / 65535;
    for (uint64_t d = 0; d < 65536; ++d)
        for (int sign = 0; sign < 2; ++sign) {
            const int64_t k = (int64_t)base + (sign ? -(int64_t)d : (int64_t)d);
            if (k <= 0 || k > 0xFFFFFFFFLL) continue;
            bool ok = true;
            for (uint32_t x = 0; x < 65535 && ok; ++x)
                ok = (uint32_t)(((uint64_t)x * (uint64_t)k) >> 32) == want[x];
            if (ok) return (uint32_t)k;
        }
    return 0;   // not reached for n <= 18 (checked by the EvoLife GPU tests)
}

// The crossover advances the RNG once for the start gene and once (twice
// with mutation) per gene: 19 or 37 applications of x -> (58321 x + 11113)
// mod 65535, composed into one affine map.  For every 16-bit x the composed
// a x + c stays below 2^32 (a, c < 65535).
static void evo_jump(EvoParams &p)
{
    const uint64_t m = 65535;
    uint64_t a = 1, c = 0;
    const int steps = 1 + 18 * (p.mutation ? 2 : 1);
    for (int k = 0; k < steps; ++k) {
        a = (58321 * a) % m;
        c = (58321 * c + 11113) % m;
    }
    p.jump_a = (uint32_t)a;
    p.jump_c = (uint32_t)c;
}

static std::once_flag g_evo_once;
static uint32_t g_evo_k[9], g_evo_kstart;

static void evo_draws(EvoParams &p, float mut_thresh)
{
    std::call_once(g_evo_once, [] {
        g_evo_k[0] = 0;
        for (uint32_t n = 1; n <= 8; ++n) g_evo_k[n] = evo_find_multiplier(n);
        g_evo_kstart = evo_find_multiplier(18);
    });
    memcpy(p.kmul, g_evo_k, sizeof(p.kmul));
    p.kstart = g_evo_kstart;
    if (!(evo_u(0) <= mut_thresh)) {
        p.mut_x = -1;
        return;
    }
    uint32_t lo = 0, hi = 65534;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) / 2;
        if (evo_u(mid) <= mut_thresh) lo = mid;
        else hi = mid - 1;
    }
    p.mut_x = (int32_t)lo;
}

// ---------------------------------------------------------------------------
// crossover tables

struct EvoDraws {
    uint32_t kmul[9], kstart;
};

// the draws of every (x0, n): thread t = x0 + 65536 (n - 1) replays the
// crossover's from x0 -- one advance for the start gene, then per visited
// gene one advance and a parent draw (and one more advance with mutation).
// Of the winner of gene g, bit 0 is bit 9 + g of .x, bit 1 bit 9 + g of .y
// (where a cell's low word holds its gene g); bit 2 is bit g of .x for g < 9,
// bit g - 9 of .y for the others; the start gene is in bits 27 .. 29 of .y.
__global__ void xk_k_evo_won(uint2 *__restrict__ won, EvoDraws d, int mutation)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 65536u * 8u) return;
    const uint32_t x0 = t & 65535u, n = (t >> 16) + 1u;
    uint32_t x = xk_lcg(x0);
    const uint32_t start = __umulhi(x, d.kstart) % 8u;
    uint2 w = make_uint2(0u, start << 27);
    for (uint32_t j = 0; j < 18; ++j) {
        x = xk_lcg(x);
        const uint32_t win = __umulhi(x, d.kmul[n]);      // < n for every state
        const uint32_t gene = start + j < 18u ? start + j : start + j - 18u;
        w.x |= (win & 1u) << (9u + gene);
        w.y |= (win >> 1 & 1u) << (9u + gene);
        if (gene < 9u) w.x |= (win >> 2) << gene;
        else w.y |= (win >> 2) << (gene - 9u);
        if (mutation) x = xk_lcg(x);
    }
    won[t] = w;
}

#define XK_EVO_TX 64            // cells of a tile; a half warp a row, four cells a lane
#define XK_EVO_TY 16
#define XK_EVO_QX (XK_EVO_TX / 4 + 2)       // quads of a row with the halo

// Byte offsets of the parents' cells in the tile, from the cell above and to
// the left of the cell, for every mask of parents (bit k: neighbour k): eight
// slots of 16 bits in neighbour order, those past the last parent the first's
__global__ void xk_k_evo_slots(uint4 *__restrict__ slots)
{
    const uint32_t pmask = threadIdx.x;
    if (pmask >= 256u) return;
    uint32_t off[8], n = 0;
    for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t c = k + (k > 3u);        // of the 3 x 3, column by column
        if (pmask >> k & 1u) off[n++] = 4u * (c % 3u * 4u * XK_EVO_QX + c / 3u);
    }
    for (uint32_t k = n; k < 8; ++k) off[k] = n != 0 ? off[0] : 0u;
    slots[pmask] = make_uint4(off[0] | off[1] << 16, off[2] | off[3] << 16, off[4] | off[5] << 16,
                              off[6] | off[7] << 16);
}

// mutation flips of every x0 (genes whose second draw is <= mut_x), in
// gene order
__global__ void xk_k_evo_mut(uint32_t *__restrict__ mut, int32_t mut_x, uint32_t kstart)
{
    const uint32_t x0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (x0 >= 65536u) return;
    uint32_t x = xk_lcg(x0);
    const uint32_t start = __umulhi(x, kstart) % 8u;
    uint32_t m = 0;
    for (uint32_t j = 0; j < 18; ++j) {
        x = xk_lcg(xk_lcg(x));
        const uint32_t gene = start + j < 18u ? start + j : start + j - 18u;
        m |= (uint32_t)((int32_t)x <= mut_x) << gene;
    }
    mut[x0] = m;
}

namespace {
struct EvoTables {
    float4 *hues = nullptr;
    uint4 *slots = nullptr;
    uint2 *won[2] = {nullptr, nullptr};        // without / with mutation
    std::map<int32_t, uint32_t *> mut;        // per mut_x
};
std::mutex g_evo_tab_mu;
std::map<std::pair<int, unsigned long long>, EvoTables> g_evo_tabs;   // per device and context
}  // namespace

// the tables for p's draws, built on first use in this device context (the
// stream is synchronised once so that every stream may use them)
static cudaError_t evo_tables(EvoParams &p, cudaStream_t s)
{
    std::lock_guard<std::mutex> lk(g_evo_tab_mu);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    EvoTables &t = g_evo_tabs[std::make_pair(dev, xk_context_id())];
    EvoDraws d;
    memcpy(d.kmul, p.kmul, sizeof(d.kmul));
    d.kstart = p.kstart;
    bool built = false;
    if (!t.hues) {
        if ((e = cudaMalloc(&t.hues, 360 * sizeof(float4))) != cudaSuccess) {
            t.hues = nullptr;
            return e;
        }
        xk_k_evo_hues<<<2, 192, 0, s>>>(t.hues);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        built = true;
    }
    p.hues = t.hues;
    if (!t.slots) {
        if ((e = cudaMalloc(&t.slots, 256 * sizeof(uint4))) != cudaSuccess) {
            t.slots = nullptr;
            return e;
        }
        xk_k_evo_slots<<<1, 256, 0, s>>>(t.slots);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        built = true;
    }
    p.slots = t.slots;
    uint2 *&won = t.won[p.mutation ? 1 : 0];
    if (!won) {
        if ((e = cudaMalloc(&won, 65536u * 8u * sizeof(uint2))) != cudaSuccess) {
            won = nullptr;
            return e;
        }
        xk_k_evo_won<<<65536u * 8u / 256u, 256, 0, s>>>(won, d, p.mutation);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        built = true;
    }
    p.won = won;
    p.mut = nullptr;
    if (p.mutation) {
        auto it = t.mut.find(p.mut_x);
        if (it == t.mut.end()) {
            uint32_t *m = nullptr;
            if ((e = cudaMalloc(&m, 65536u * sizeof(uint32_t))) != cudaSuccess) return e;
            xk_k_evo_mut<<<65536u / 256u, 256, 0, s>>>(m, p.mut_x, p.kstart);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
            it = t.mut.emplace(p.mut_x, m).first;
            built = true;
        }
        p.mut = it->second;
    }
    return built ? cudaStreamSynchronize(s) : cudaSuccess;
}

#define XK_EVO_MINB 4           // 64 registers

struct __align__(16) EvoTile {
    uint32_t lo[XK_EVO_TY + 2][4 * XK_EVO_QX];      // low words of the cells: column c at c + 4
    uint2 ma[XK_EVO_TY + 2][XK_EVO_QX];             // per quad: birth bits, living cells, a byte a cell
    uint4 slots[256];                               // EvoParams::slots
    float4 hues[360];                               // EvoParams::hues
    int4 col[XK_EVO_TY][xk_col_pieces(XK_EVO_TX)];  // colours (frame.cuh)
};

// bits of a where m is set, else of b
__device__ __forceinline__ uint32_t xk_evo_mux(uint32_t m, uint32_t a, uint32_t b) { return (a & m) | (b & ~m); }

// A quad of cells into the tile
__device__ __forceinline__ void xk_evo_put(EvoTile &T, int r, int qx, const uint64_t v[4])
{
    uint32_t lo[4], alive[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        lo[k] = (uint32_t)v[k];
        alive[k] = min(lo[k] & 0x7FFFFFFu, 1u);         // xmath.min(1, energy + rule)
    }
    *(uint4 *)&T.lo[r][4 * qx] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    // birth bits: bits 10 .. 17 of a cell
    const uint32_t a = __byte_perm(lo[0], lo[1], 0x6521) >> 2, b = __byte_perm(lo[2], lo[3], 0x6521) >> 2;
    T.ma[r][qx] = make_uint2(__byte_perm(a, b, 0x6420),
                             alive[0] + alive[1] * 256u + alive[2] * 65536u + alive[3] * 16777216u);
}

// What the crossover's genome makes of a cell (its low word lo, `alive` living
// neighbours, random state `state`): the reference's selections by
// multiplication as selects (the same integers).  A new genome replaces the
// rule and resets the energy, a cell that does not live keeps neither; the
// crossover advances the random state by the composed map.
__device__ __forceinline__ uint64_t xk_evo_cell(const EvoParams &p, uint32_t lo, uint32_t state, uint32_t alive,
                                                uint32_t genome, uint32_t &rule, uint32_t &energy)
{
    const uint32_t old_energy = lo & 511u, old_rule = lo >> 9 & 262143u;
    const uint32_t sustained = (old_rule & 261120u) >> (alive + 9u) & 1u;
    rule = genome != 0 ? genome : old_rule;
    const bool is_live = old_energy < 255u && ((lo & 0x7FFFFFFu) == 0u || sustained != 0u);
    const uint32_t new_energy = old_energy + ((lo & 0x7FFFFFFu) != 0u ? p.death_speed : 0u);
    energy = rule == old_rule && is_live ? (uint16_t)new_energy : 0u;
    rule = is_live ? rule : 0u;
    const uint32_t rng = (p.jump_a * state + p.jump_c) % 65535u;
    return (uint64_t)((energy & 511u) | rule << 9) | (uint64_t)rng << 27;
}

// Four cells of a row from column x; W is a multiple of 4, so quads wrap whole
__device__ __forceinline__ void xk_evo_get(const uint64_t *__restrict__ row, int x, int W, uint64_t v[4])
{
    if ((unsigned)x >= (unsigned)W) {
        x %= W;
        if (x < 0) x += W;
    }
    const ulonglong2 a = __ldg((const ulonglong2 *)(row + x)), b = __ldg((const ulonglong2 *)(row + x + 2));
    v[0] = a.x;
    v[1] = a.y;
    v[2] = b.x;
    v[3] = b.y;
}

// num_parents for every birth count 1..8 at once, bit-sliced, from the birth
// bits of a cell's eight neighbours (a byte a cell): lane g of the 4-bit
// counts (b3 b2 b1 b0) counts the neighbours whose rule has bit g + 1 (a dead
// neighbour has rule 0), by a carry-save tree.  The lanes with a fit: those
// whose count equals g + 1 (bit planes of g + 1 per lane: 0x55, 0x66, 0x78,
// 0x80).
__device__ __forceinline__ uint32_t xk_evo_fits(const uint32_t m[8])
{
    const uint32_t s0 = m[0] ^ m[1] ^ m[2], c0 = (m[0] & m[1]) | (m[2] & (m[0] ^ m[1]));
    const uint32_t s1 = m[3] ^ m[4] ^ m[5], c1 = (m[3] & m[4]) | (m[5] & (m[3] ^ m[4]));
    const uint32_t s2 = m[6] ^ m[7], c2 = m[6] & m[7];
    const uint32_t b0 = s0 ^ s1 ^ s2, c3 = (s0 & s1) | (s2 & (s0 ^ s1));
    const uint32_t t0 = c0 ^ c1 ^ c2, d0 = (c0 & c1) | (c2 & (c0 ^ c1));
    const uint32_t b1 = t0 ^ c3, d1 = t0 & c3;
    const uint32_t b2 = d0 ^ d1, b3 = d0 & d1;
    return (b0 ^ 0xAAAAAAAAu) & (b1 ^ 0x99999999u) & (b2 ^ 0x87878787u) & (b3 ^ 0x7F7F7F7Fu);
}

// One cell a thread, neighbours read from global memory: rows that do not
// start on 16-byte boundaries, and lattices whose quads are too few to fill
// the chip (xk_evolife_step's rule).
template <bool MUT>
__global__ void __launch_bounds__(256, 8)
xk_k_evolife_one(const uint64_t *__restrict__ src, uint64_t *__restrict__ dst, int32_t *__restrict__ col,
                 EvoParams p)
{
    const int x = blockIdx.x * 32 + threadIdx.x;
    const int y = blockIdx.y * 8 + threadIdx.y;
    if (x >= p.W || y >= p.H) return;   // no block-wide synchronisation below
    xk_grid_dep_wait();                 // launched as a dependent of the previous generation
    const int xl = x > 0 ? x - 1 : p.W - 1, xr = x < p.W - 1 ? x + 1 : 0;
    const int yu = y > 0 ? y - 1 : p.H - 1, yd = y < p.H - 1 ? y + 1 : 0;
    const int nxs[8] = {xl, xl, xl, x, x, xr, xr, xr};
    const int nys[8] = {yu, y, yd, yu, yd, yu, y, yd};
    // a neighbour's energy (bits 0-8) and rule (bits 9-26) are both in the
    // low 32-bit half of its cell: only that half is read
    const uint32_t *src_lo = reinterpret_cast<const uint32_t *>(src);
    uint32_t nlo[8], m[8], alive = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        nlo[k] = __ldg(src_lo + 2 * ((int64_t)nys[k] * p.W + nxs[k]));
        alive += (nlo[k] & 0x7FFFFFFu) != 0u;   // xmath.min(1, e + r): e + r != 0
        m[k] = nlo[k] >> 10 & 255u;
    }
    const int64_t i = (int64_t)y * p.W + x;
    const uint64_t c = src[i];
    const uint32_t state = (uint32_t)(c >> 27) & 65535u;
    const uint32_t n = 32u - (uint32_t)__clz(xk_evo_fits(m) & 255u);
    uint32_t genome = 0;
    if (n != 0) {
        const uint2 won = __ldg(p.won + (65536u * (n - 1u) + state));
        // the planes of the winner's slot, less the parents passed: zero
        // where the next parent wins
        uint32_t b0 = won.x, b1 = won.y, b2 = (won.x & 511u) << 9 | (won.y & 511u) << 18, g = 0, any = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (m[k] >> (n - 1u) & 1u) {
                g |= nlo[k] & ~(b0 | b1 | b2);
                any |= nlo[k];
                b2 ^= ~(b0 | b1);
                b1 ^= ~b0;
                b0 = ~b0;
            }
        genome = g >> 9 & 262143u;
        int excess = __popc(genome) - (int)p.max_genes;
        if (excess > 0) {
            const uint32_t start = won.y >> 27;
            uint32_t rot = xk_rot18(genome, start);
            do rot &= ~(0x80000000u >> __clz(rot));
            while (--excess > 0);
            genome = xk_unrot18(rot, start);
        }
        if (MUT) genome ^= __ldg(p.mut + state) & (any >> 9);
    }
    uint32_t rule, energy;
    const uint64_t out = xk_evo_cell(p, (uint32_t)c, state, alive, genome, rule, energy);
    if (p.color_kind != XK_COLOR_NONE) {
        const int3 v = p.positional ? xk_evo_color_positional(rule, energy)
                                    : xk_evo_color_modular(p.hues, rule, energy);
        int rgb[3] = {v.x, v.y, v.z};
        if (p.color_kind == XK_COLOR_MOVING_AVERAGE)
#pragma unroll
            for (int ch = 0; ch < 3; ++ch)
                rgb[ch] = xk_fade(rgb[ch] * p.smooth, col[3 * i + ch], p.fade_in, p.neg_fade_out);
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) col[3 * i + ch] = rgb[ch];
        if (p.frame)
#pragma unroll
            for (int ch = 0; ch < 3; ++ch)
                p.frame[3 * i + ch] = (uint8_t)(p.small ? (uint32_t)rgb[ch] : xk_pixel(rgb[ch], p.frame_smooth));
    }
    dst[i] = out;
}

// Four cells a thread, rows of a multiple of four cells.  MUT: mutation_prob >
// 0 (the mutation flips, and the union of the parents' genomes they are masked
// with, exist only then).  POS: the positional genome colour.
template <bool MUT, bool POS>
__global__ void __launch_bounds__(256, XK_EVO_MINB)
xk_k_evolife(const uint64_t *__restrict__ src, uint64_t *__restrict__ dst, int32_t *__restrict__ col,
             EvoParams p)
{
    __shared__ EvoTile T;
    const int tid = threadIdx.x, lane = tid & 31, q = tid & 15, r = tid >> 4;
    const int by = blockIdx.x / p.tiles_x, bx = blockIdx.x - by * p.tiles_x;
    const int x0 = bx * XK_EVO_TX, y0 = by * XK_EVO_TY;
    const int x = x0 + 4 * q, y = y0 + r;
    const bool row_in = y < p.H, in = row_in && x < p.W;
    const int width = min(XK_EVO_TX, p.W - x0);
    const int64_t i = (int64_t)y * p.W + x;
    xk_grid_dep_wait();                 // launched as a dependent of the previous generation
    const bool fades = p.color_kind == XK_COLOR_MOVING_AVERAGE;
    const int64_t first = 3 * ((int64_t)y * p.W + x0);      // the row's first colour word
    if (fades && row_in)
        xk_col_fetch<XK_EVO_TX>(T.col[r], col, first, width, q);
    xk_copy_async16(&T.slots[tid], p.slots + tid);
    if (!POS)
        for (int k = tid; k < 360; k += 256) xk_copy_async16(&T.hues[k], p.hues + k);
    uint64_t own[4], halo[4];
    xk_evo_get(src + (int64_t)(row_in ? y : y % p.H) * p.W, x, p.W, own);
    const int h = tid - 2 * XK_EVO_QX;              // the halo: two rows, then two quads a row
    const int hr = h >= 0 ? 1 + (h >> 1) : tid < XK_EVO_QX ? 0 : XK_EVO_TY + 1;
    const int hq = h >= 0 ? (h & 1) * (XK_EVO_QX - 1) : tid < XK_EVO_QX ? tid : tid - XK_EVO_QX;
    const bool rim = h < 2 * XK_EVO_TY;
    if (rim) {
        int gy = y0 + hr - 1;
        if (gy < 0) gy += p.H;
        else if (gy >= p.H) gy %= p.H;
        xk_evo_get(src + (int64_t)gy * p.W, x0 + 4 * hq - 4, p.W, halo);
    }
    xk_evo_put(T, r + 1, q + 1, own);
    if (rim) xk_evo_put(T, hr, hq, halo);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    // the eight neighbours' birth bits as words of four cells, in neighbour
    // order; living neighbours by column sums
    uint32_t m[8], alive;
    {
        const uint2 *u = &T.ma[r][q], *c = &T.ma[r + 1][q], *d = &T.ma[r + 2][q];
        const uint2 ul = u[0], uc = u[1], ur = u[2], cl = c[0], cc = c[1], cr = c[2], dl = d[0], dc = d[1], dr = d[2];
        m[0] = __byte_perm(ul.x, uc.x, 0x6543);
        m[1] = __byte_perm(cl.x, cc.x, 0x6543);
        m[2] = __byte_perm(dl.x, dc.x, 0x6543);
        m[3] = uc.x;
        m[4] = dc.x;
        m[5] = __byte_perm(uc.x, ur.x, 0x4321);
        m[6] = __byte_perm(cc.x, cr.x, 0x4321);
        m[7] = __byte_perm(dc.x, dr.x, 0x4321);
        const uint32_t l = ul.y + cl.y + dl.y, ud = uc.y + dc.y, mid = ud + cc.y, rt = ur.y + cr.y + dr.y;
        alive = ud + __byte_perm(l, mid, 0x6543) + __byte_perm(mid, rt, 0x4321);
    }
    const uint32_t eq = xk_evo_fits(m);
    // parents: rules with the largest fitting birth count (num_fit, their
    // number), in neighbour order.  A cell's eight birth bytes in two words;
    // bit num_fit - 1 of each gathered into a mask by byte dot products.
    uint32_t n[4], pmask[4];
    uint2 won[4];
    {
        uint32_t near[4], far[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t *o = h ? far : near;
            const uint32_t a = __byte_perm(m[4 * h], m[4 * h + 1], 0x5140),
                           b = __byte_perm(m[4 * h], m[4 * h + 1], 0x7362),
                           c = __byte_perm(m[4 * h + 2], m[4 * h + 3], 0x5140),
                           d = __byte_perm(m[4 * h + 2], m[4 * h + 3], 0x7362);
            o[0] = __byte_perm(a, c, 0x5410);
            o[1] = __byte_perm(a, c, 0x7632);
            o[2] = __byte_perm(b, d, 0x5410);
            o[3] = __byte_perm(b, d, 0x7632);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            n[k] = 32u - (uint32_t)__clz(eq >> (8 * k) & 255u);
            const uint32_t f = max(n[k], 1u) - 1u;      // (none: what one parent would win, cleared below)
            const uint32_t state = (uint32_t)(own[k] >> 27) & 65535u;
            won[k] = make_uint2(0, 0);
            if (n[k] != 0) won[k] = __ldg(p.won + (65536u * f + state));
            pmask[k] = __dp4a(near[k] >> f & 0x01010101u, 0x08040201u, 0u);
            pmask[k] = __dp4a(far[k] >> f & 0x01010101u, 0x80402010u, pmask[k]);
        }
    }
    int *mine = (int *)T.col[r] + 12 * q;
    int c[12];
    if (fades) xk_col_read(mine, c);
    // genome_crossover(main, 18, *genomes, max_genes, mutation_prob), step by
    // step for the four cells.  With no parent, every gene is 0 (no winner,
    // and a mutation needs a gene that some parent has).
    uint32_t genome[4], any[4];
    const uint32_t most = max(max(n[0], n[1]), max(n[2], n[3]));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const char *at = (const char *)&T.lo[r][4 * q + 3 + k];
        auto slot = [&](uint32_t o) { return *(const uint32_t *)(at + o); };
        uint4 s = make_uint4(0, 0, 0, 0);
        if (n[k] > 0) s = T.slots[pmask[k]];
        uint32_t p0 = 0, p1 = 0, p2 = 0, p3 = 0;
        if (n[k] > 0) p0 = slot(s.x & 65535u);
        if (n[k] > 1) p1 = slot(s.x >> 16);
        if (n[k] > 2) p2 = slot(s.y & 65535u);
        if (n[k] > 3) p3 = slot(s.y >> 16);
        uint32_t g = xk_evo_mux(won[k].y, xk_evo_mux(won[k].x, p3, p2), xk_evo_mux(won[k].x, p1, p0));
        any[k] = p0 | p1 | p2 | p3;
        if (most > 4) {
            uint32_t p4 = 0, p5 = 0, p6 = 0, p7 = 0;
            if (n[k] > 4) p4 = slot(s.z & 65535u);
            if (n[k] > 5) p5 = slot(s.z >> 16);
            if (n[k] > 6) p6 = slot(s.w & 65535u);
            if (n[k] > 7) p7 = slot(s.w >> 16);
            any[k] |= p4 | p5 | p6 | p7;
            g = xk_evo_mux((won[k].x & 511u) << 9 | (won[k].y & 511u) << 18,
                           xk_evo_mux(won[k].y, xk_evo_mux(won[k].x, p7, p6), xk_evo_mux(won[k].x, p5, p4)), g);
        }
        genome[k] = g >> 9 & 262143u;
        any[k] >>= 9;
    }
    // the first max_genes genes taken, in visiting order (from the start
    // gene, wrapping at 18): the last ones of the word rotated to it go
    int excess[4], longest = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        excess[k] = __popc(genome[k]) - (int)p.max_genes;
        longest = max(longest, excess[k]);
    }
    if (longest > 0) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t start = won[k].y >> 27;
            genome[k] = xk_rot18(genome[k], start);
        }
        do {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (excess[k] > 0) genome[k] &= ~(0x80000000u >> __clz(genome[k]));
                --excess[k];
            }
        } while (--longest > 0);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t start = won[k].y >> 27;
            genome[k] = xk_unrot18(genome[k], start);
        }
    }
    uint64_t out[4];
    uint32_t rules[4], energies[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t state = (uint32_t)(own[k] >> 27) & 65535u;
        if (MUT) genome[k] ^= __ldg(p.mut + state) & any[k];
        out[k] = xk_evo_cell(p, (uint32_t)own[k], state, alive >> (8 * k) & 255u, genome[k], rules[k], energies[k]);
    }
    if (p.color_kind != XK_COLOR_NONE)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int3 v = POS ? xk_evo_color_positional(rules[k], energies[k])
                                        : xk_evo_color_modular(T.hues, rules[k], energies[k]);
            c[3 * k] = fades ? xk_fade(v.x * p.smooth, c[3 * k], p.fade_in, p.neg_fade_out) : v.x;
            c[3 * k + 1] = fades ? xk_fade(v.y * p.smooth, c[3 * k + 1], p.fade_in, p.neg_fade_out) : v.y;
            c[3 * k + 2] = fades ? xk_fade(v.z * p.smooth, c[3 * k + 2], p.fade_in, p.neg_fade_out) : v.z;
        }
    if (in)
        asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(dst + i), "l"(out[0]), "l"(out[1]),
                     "l"(out[2]), "l"(out[3])
                     : "memory");
    if (p.color_kind == XK_COLOR_NONE) return;
    xk_col_write(mine, c);
    __syncwarp();
    if (row_in) xk_col_store<XK_EVO_TX>(T.col[r], col, first, width, q);
    if (!p.frame) return;
    uint32_t b[3];
    xk_pixels4(c, mine, p.small != 0, p.frame_smooth, b);
    const int left = lane & 16;                     // the row's half warp
    xk_store_px4(p.frame + 3 * i, b, lane, left, row_in ? left + width / 4 - 1 : -1);
}

cudaError_t xk_evolife_set_positional(const double *lut54)
{
    return cudaMemcpyToSymbol(c_evo_pos, lut54, 54 * sizeof(double));
}

cudaError_t xk_evolife_step(const uint64_t *src, uint64_t *dst, int32_t *col, const xk_desc &d,
                            float mut_thresh, const int32_t *col_range, cudaStream_t s, uint8_t *frame,
                            int frame_smooth)
{
    EvoParams p;
    p.W = (int32_t)d.size[0];
    p.H = (int32_t)d.size[1];
    p.death_speed = d.death_speed;
    p.max_genes = d.max_genes;
    p.mutation = d.mutation_prob > 0.0;
    p.positional = d.positional;
    p.color_kind = d.color_kind;
    p.fade_in = d.fade_in;
    p.neg_fade_out = (int32_t)(0u - (uint32_t)d.fade_out);
    p.smooth = d.smooth;
    p.frame = frame;
    p.frame_smooth = frame_smooth;
    p.small = xk_px_stays_small(d, frame_smooth) && xk_px_small(col_range[0]) && xk_px_small(col_range[1]);
    evo_draws(p, mut_thresh);
    evo_jump(p);
    cudaError_t e = evo_tables(p, s);
    if (e != cudaSuccess) return e;
    // Four cells a thread from 3 * 2^18 cells, where they fill the chip, in
    // rows of a multiple of four: 64 generations with frames take 746 us of
    // them and 800 one a thread at 1280 x 720 (531 and 498 at 800 x 600, 257
    // and 190 at 320 x 200); with quads cut to words and bytes at 1919 x 1079
    // 1830 and 1626.
    if (p.W % 4 != 0 || !xk_tiles_in_range(p.W, p.H) || (int64_t)p.W * p.H < 3 << 18) {
        const dim3 block(32, 8), grid((p.W + 31) / 32, (p.H + 7) / 8);
        return p.mutation ? xk_launch_pdl(xk_k_evolife_one<true>, grid, block, 0, s, src, dst, col, p)
                          : xk_launch_pdl(xk_k_evolife_one<false>, grid, block, 0, s, src, dst, col, p);
    }
    p.tiles_x = (p.W + XK_EVO_TX - 1) / XK_EVO_TX;
    const dim3 block(256), grid(p.tiles_x * ((p.H + XK_EVO_TY - 1) / XK_EVO_TY));
    auto run = [&](auto kernel) { return xk_launch_pdl(kernel, grid, block, 0, s, src, dst, col, p); };
    if (p.mutation) return p.positional ? run(xk_k_evolife<true, true>) : run(xk_k_evolife<true, false>);
    return p.positional ? run(xk_k_evolife<false, true>) : run(xk_k_evolife<false, false>);
}
