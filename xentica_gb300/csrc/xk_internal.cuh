// Internal declarations shared by the libxk translation units.
#pragma once

#include <stdlib.h>
#include <string.h>

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string>
#include <vector>

#include "../../include/xk.h"

// ---------------------------------------------------------------------------
// error handling: every C-ABI function returns a status and records a message
void xk_set_error(const char *fmt, ...);
int xk_cuda_status(cudaError_t err, const char *what);

#define XK_CUDA(call)                                                         \
    do {                                                                      \
        cudaError_t xk_e_ = (call);                                           \
        if (xk_e_ != cudaSuccess) return xk_cuda_status(xk_e_, #call);        \
    } while (0)

#define XK_REQUIRE(cond, code, ...)                                           \
    do {                                                                      \
        if (!(cond)) { xk_set_error(__VA_ARGS__); return (code); }            \
    } while (0)

void xk_set_last_step_ms(double ms);

// ---------------------------------------------------------------------------
// Life-like bit-packed lattices: cell x of row y is bit (x & 31) of word
// y * wpr + (x >> 5); padding bits past the row's last cell are always 0.

// The rule as the coefficients of the multiplexer tree's first level.  The
// truth-table masks T[s][n] (0 or ~0: the next state of a cell in state s
// with n live neighbours) are paired by the count's bit 0, and
// `sel ? B : A` over masks A, B is the integer multiply-add sel * k + A with
// k = 0 (A == B), 1 (A = 0, B = ~0) or ~0 (A = ~0, B = 0), exactly, on the
// FMA pipe instead of the logic pipe.  Pair q < 4: A = T[0][2q],
// B = T[0][2q + 1]; q >= 4: the same for T[1][2(q - 4)].  a8/k8: the count-8
// pair (T[0][8], T[1][8]) selected by the cell's state.
struct LifeTable {
    uint32_t a[8], k[8];
    uint32_t a8, k8;
};

// The same rule over the count n9 of the 3 x 3 block including the cell
// (0..9; a live cell's n9 is its neighbour count + 1): dead D[n] = T[0][n],
// live L[n] = T[1][n - 1] (L[0] never occurs and repeats L[1]).  Pairs by
// the count's bit 0: q < 4 (D[2q], D[2q + 1]), q >= 4 (L[2(q - 4)],
// L[2(q - 4) + 1]); n9 of 8 or 9: D[8] for a dead cell, the pair (L[8], L[9])
// (a9, k9) for a live one.
struct LifeTable9 {
    uint32_t a[8], k[8];
    uint32_t d8, a9, k9;
};

__host__ __device__ inline uint32_t xk_mux_coef(uint32_t A, uint32_t B)
{
    return A == B ? 0u : (A ? 0xFFFFFFFFu : 1u);
}

LifeTable xk_life_table(uint32_t rule0, uint32_t rule1);

struct LifeGeo {
    int32_t W, H, wpr, rlast;  // width, height, words per row, bits in last word
    uint32_t lastmask;         // valid bits of a row's last word
    int32_t torus;             // 1: wrap; 0: off-board cells read as bfill
    uint32_t bfill;            // 0 or ~0: static border state replicated
    uint32_t div_wpr;          // xk_div_magic(wpr, H * wpr)
};

// n / d for every n < N as umulhi(n, m) with m = ceil(2^32 / d): exact when
// N * (m d - 2^32) < 2^32 (then n / d + n e / (d 2^32) stays below the next
// integer); 0 when that does not hold or d < 2, meaning a plain division
inline uint32_t xk_div_magic(uint64_t d, uint64_t N)
{
    if (d < 2 || d >= (1ull << 32)) return 0;
    const uint64_t m = ((1ull << 32) + d - 1) / d;
    const uint64_t e = m * d - (1ull << 32);
    return (e == 0 || N < (1ull << 32) / e) && N <= 0xFFFFFFFFull ? (uint32_t)m : 0u;
}

__device__ __forceinline__ uint32_t xk_divu(uint32_t n, uint32_t d, uint32_t m)
{
    return m ? __umulhi(n, m) : n / d;
}

// 16-cell halves that word j of a row of W cells holds, W a multiple of 16
// (unsigned: the words of the widest row end at 2^31)
__host__ __device__ __forceinline__ int xk_word_halves(uint32_t j, int32_t W)
{
    return 32u * j + 32u <= (uint32_t)W ? 2 : 1;
}

// Column of a torus row that x stands for, a column outside it: up to 2^29
// beyond its end, or before its start (2^32 less the distance)
__host__ __device__ __forceinline__ int xk_wrap_column(uint32_t x, int W)
{
    const int c = (int)(x < 0xC0000000u ? x - (uint32_t)W : x) % W;
    return c < 0 ? c + W : c;
}

// Whether the coordinates of tiles of up to 64 cells a side, their halo and
// the cells loaded beside it (64 in all beyond the last cell) are 32-bit ints
__host__ __device__ constexpr bool xk_tiles_in_range(int64_t W, int64_t H)
{
    return W <= 0x7FFFFFFFll - 64 && H <= 0x7FFFFFFFll - 64;
}

LifeGeo xk_life_geo(int64_t W, int64_t H, int torus, int border_state);

// one lattice (or ensemble instance) for the resident kernel
struct LifeInst {
    int64_t off;               // first word in the state array
    int32_t W, H, wpr, rlast;
    uint32_t lastmask;
    uint32_t rule0, rule1;
    int32_t smem_words;        // shared memory the instance needs
};

// shared-memory words a resident lattice needs with `threads` threads
int64_t xk_life_resident_words(int W, int H, int threads);
// largest dynamic shared memory a CTA may use on this device
int xk_max_smem_optin();
// identity of the CUDA context current on this thread (unique for the
// process's lifetime; 0 when it cannot be told): device-side objects cached
// per context are looked up again after a context reset
unsigned long long xk_context_id();
// Raise a kernel's cudaFuncAttributeMaxDynamicSharedMemorySize (one value per
// function and device) to at least `bytes`; never lowers it.  A graph node
// keeps the shared memory of the launch it captured, and a node launched or
// replayed later (a profiler replays graph nodes one by one) is checked
// against the attribute as it is then: had a later, smaller launch lowered
// the attribute, that node would fail with cudaErrorLaunchFailure or an
// invalid-argument error.  Kept monotone, every captured node stays valid.
cudaError_t xk_smem_attr_at_least(const void *fn, int bytes);

// launchers (stream-ordered, no synchronisation)
cudaError_t xk_life_pack(const void *src, int esz, uint32_t *dst, const LifeGeo &g, cudaStream_t s);
cudaError_t xk_life_unpack(const uint32_t *src, void *dst, int esz, const LifeGeo &g, cudaStream_t s);
cudaError_t xk_life_step_global(const uint32_t *src, uint32_t *dst, const LifeGeo &g,
                                const LifeTable &t, cudaStream_t s);
// bytes_io: state is one byte per cell (LifeInst.off in bytes) instead of
// bit-packed words; `bad` (bytes_io only) is or-ed with 1 if a cell held a
// value other than 0/1
// rule_form (bit-packed state only): XK_RULE_CONWAY runs the instantiation
// with B3/S23 compiled in (every instance's rule must then be B3/S23)
// priority (one-byte torus state only): the launch's priority attribute
// (a graph instantiated with cudaGraphInstantiateFlagUseNodePriority keeps it)
#define XK_NO_PRIORITY (-1000000)
cudaError_t xk_life_step_resident(const LifeInst *inst, int ninst, void *state, int bytes_io,
                                  int generations, int torus, uint32_t bfill, unsigned int *bad,
                                  int threads, int smem_bytes, cudaStream_t s, int rule_form = 0,
                                  int priority = XK_NO_PRIORITY);
// torus, one byte per cell, in place: lattice k advances gens[k]
// generations (a device array of ninst counts)
cudaError_t xk_life_step_resident_each(const LifeInst *inst, const int32_t *gens, int ninst, void *state,
                                       unsigned int *bad, int threads, int smem_bytes, cudaStream_t s);
// torus, one byte per cell: lattices read from `in`, results written to
// `out` and, when `mirror` is not null, also to `mirror` (the same offsets);
// `in` and `out` may be device addresses of mapped host memory
cudaError_t xk_life_step_resident_io(const LifeInst *inst, int ninst, const uint8_t *in, uint8_t *out,
                                     uint8_t *mirror, int generations, unsigned int *bad, int threads,
                                     int smem_bytes, cudaStream_t s);
// CTAs of that kernel one SM holds at once with this block size and
// shared memory (1 when the query fails)
int xk_life_resident_ctas_per_sm(int threads, int smem_bytes);
// threads and dynamic shared memory of the resident kernel for one lattice;
// rows_per_band: target band length (controls the number of warps)
int xk_life_resident_config(int W, int H, int rows_per_band, int *threads, int *smem_bytes);
cudaError_t xk_life_colors(const uint32_t *bits, int32_t *col, const LifeGeo &g,
                           const int32_t *lut6, int smooth, cudaStream_t s);
cudaError_t xk_life_color_step(const uint32_t *bits, int32_t *col, const LifeGeo &g,
                               const int32_t *lut6, int fade_in, int fade_out, int smooth,
                               int plain, cudaStream_t s);

// 3-D von Neumann Life-like, bit-packed along x; row (y, z) is row z * H + y
// (pack/unpack with xk_life_geo(W, H * D, torus, border state))
struct Life3Geo {
    int32_t W, H, D, wpr, rlast;
    uint32_t lastmask;
    uint32_t div_wpr, div_h;   // xk_div_magic(wpr, H * D * wpr), xk_div_magic(H, H * D)
    int32_t torus;
    uint32_t bfill;            // static border: its state in every bit
};
// (div_h only for lattices of fewer than 2^32 words, which the kernels take)
Life3Geo xk_life3_geo(int64_t W, int64_t H, int64_t D, int torus, int border_state);
cudaError_t xk_life_step3d_vn(const uint32_t *src, uint32_t *dst, const Life3Geo &g,
                              const LifeTable &t, cudaStream_t s);
// the same on a cluster of C CTAs that hold the lattice, in place
// (life3d_cluster.cu); plan returns 0 when it does not fit one
struct Life3ClPlan {
    int C, most, smem;         // CTAs, planes of the largest slab, dynamic shared memory
};
int xk_life3d_cluster_plan(const Life3Geo &g, bool alone, Life3ClPlan *out);
cudaError_t xk_life_step3d_cluster(uint32_t *cells, const Life3Geo &g, const LifeTable &t, int generations,
                                   const Life3ClPlan &p, cudaStream_t s);

// one lattice (W <= 1024) on a thread-block cluster of C CTAs, R rows each,
// in place on its bit-packed words (cluster.cu); config returns 0 when no
// cluster of (up to) C CTAs whose lane groups walk bands of about `band` rows
// fits
LifeTable9 xk_life_table9(uint32_t rule0, uint32_t rule1);
// Rule forms of the single-lattice kernels: a rule loaded at run time, or
// Conway's Life B3/S23 fixed at compile time (the reference's default
// LifelikeCA rule and its GameOfLife model)
#define XK_RULE_TABLE 0
#define XK_RULE_CONWAY 1
// the rule form a single-lattice kernel compiles for (rule0: dead-cell table,
// rule1: live-cell table): XK_RULE_CONWAY for B3/S23, else XK_RULE_TABLE
int xk_rule_form(uint32_t rule0, uint32_t rule1);
int xk_life_cluster_config(const LifeGeo &g, int C, int band, int *C_out, int *R, int *threads);
// sync: how the CTAs of the cluster order their halo exchange every
// generation -- XK_SYNC_BARRIER a cluster barrier; XK_SYNC_NEIGHBOUR mbarriers
// of the two neighbouring CTAs only (bands of 1, 2 and 4 rows);
// XK_SYNC_SPLIT a cluster barrier whose arrive and wait enclose the bands'
// inner rows (every CTA's bands exactly 4 or 8 rows); XK_SYNC_ASYNC the
// neighbour form with the rows sent by asynchronous remote stores that
// complete a transaction count on the receiver's mbarrier (bands of 1 row, or
// every CTA's bands exactly 2, 4 or 8 rows): xk_life_cluster_has_sync
#define XK_SYNC_BARRIER 0
#define XK_SYNC_NEIGHBOUR 1
#define XK_SYNC_SPLIT 2
#define XK_SYNC_ASYNC 3
cudaError_t xk_life_step_cluster(uint32_t *bits, const LifeGeo &g, uint32_t rule0, uint32_t rule1,
                                 int generations, int C, int R, int threads, cudaStream_t s, int sync = 0);
int xk_life_cluster_has_sync(const LifeGeo &g, int C, int R, int threads, int sync);
// a CTA of the neighbour form gave up waiting since the last call (clears it)
bool xk_cluster_take_wait_failure();

// The same lattices with rows exchanged every 8 generations
// (cluster_deep.cu): config returns 0 where no cluster of (up to) C CTAs with
// B (2, 3, 4, 6) rows a lane group applies (every CTA needs 8 rows); *gave_up
// (device memory) is or-ed with 1 when a bounded wait gave up.
struct DeepPlan {
    int C = 0, R = 0, B = 0, bands = 0, threads = 0, smem = 0;
};
int xk_life_deep_config(const LifeGeo &g, int C, int B, DeepPlan *out);
cudaError_t xk_life_step_deep(uint32_t *bits, const LifeGeo &g, uint32_t rule0, uint32_t rule1, int generations,
                              const DeepPlan &p, unsigned int *gave_up, cudaStream_t s);

// T (1 .. XK_TB_DEEPEST) generations per launch of a 2-D lattice of any size
// (W >= 64), tiles with a T-generation halo in registers, src -> dst
// (life_tb.cu)
#define XK_TB_DEEPEST 12
int xk_life_tb_supported(const LifeGeo &g);
// generations of a launch of a plan of this depth (2 .. 8): a depth of 8 asks
// for as many as pay.  960 generations take 1 295 us of 12 a launch and 1 414
// of 8 at 4096 x 4096, 454 and 473 at 1100 x 1100, 554 and 574 at 2000 x 1500;
// 16 are up to 8 % slower at some sizes, 3 % faster at others.
inline int xk_life_tb_launch(int depth) { return depth == 8 ? XK_TB_DEEPEST : depth; }
cudaError_t xk_life_step_tb(const uint32_t *src, uint32_t *dst, const LifeGeo &g, const LifeTable9 &t,
                            int T, cudaStream_t s);

// byte-per-cell lattices (N-D, any neighbourhood; and the plain 2-D form)
struct NdGeo {
    int32_t ndim, nbr, torus;
    int64_t size[XK_MAXDIM];
    int8_t delta[XK_MAXNBR][XK_MAXDIM];
    uint32_t border_state;      // 0/1 state of off-board cells
};
// bit-packed along axis 0 (life_nd.cu): n / W rows of wpr words, neighbours
// grouped by row (delta[k][1..]; delta[k][0]: bit 0 the left, 1 the middle, 2
// the right cell of the row)
struct BitsNdGeo {
    int32_t ndim, nbr, groups, torus, moore3d, faces3d;
    int32_t size[XK_MAXDIM];
    int8_t delta[XK_MAXNBR][XK_MAXDIM];
    int32_t wpr, rlast;
    uint32_t lastmask, bfill;
    uint32_t words;             // rows * wpr
    uint32_t div_wpr, div_h;    // xk_div_magic(wpr, words); 3-D: xk_div_magic(size[1], rows)
};
// the rule over the neighbour count 0..31 as LifeTable's coefficients: pair
// q < 16 (dead 2q, 2q + 1), q >= 16 the same for live cells
struct LifeTable32 {
    uint32_t a[32], k[32];
};
// the bit-packed form of a lattice; 0 where its kernels do not apply (offsets
// of more than one cell, more than 2^31 words)
int xk_bits_nd_geo(const NdGeo &nd, BitsNdGeo *out);
cudaError_t xk_life_step_bits_nd(const uint32_t *src, uint32_t *dst, const BitsNdGeo &g, uint32_t rule0,
                                 uint32_t rule1, cudaStream_t s);
cudaError_t xk_nd_pack(const void *src, int esz, uint8_t *dst, int64_t n, cudaStream_t s);
cudaError_t xk_nd_unpack(const uint8_t *src, void *dst, int esz, int64_t n, cudaStream_t s);
cudaError_t xk_life_step_nd(const uint8_t *src, uint8_t *dst, const NdGeo &g, uint32_t rule0,
                            uint32_t rule1, cudaStream_t s);
cudaError_t xk_life_step_bytes2d(const uint8_t *src, uint8_t *dst, int W, int H,
                                 uint32_t rule0, uint32_t rule1, cudaStream_t s);
// shifting family (shift.cu): one generation (any topology and border), or
// `generations` at once on a torus
cudaError_t xk_shift_step_nd(const uint8_t *src, uint8_t *dst, const NdGeo &g, int i0, cudaStream_t s);
cudaError_t xk_shift_jump(const uint8_t *src, uint8_t *dst, const NdGeo &g, int i0, int64_t generations,
                          cudaStream_t s);
cudaError_t xk_nd_colors(const uint8_t *st, int32_t *col, int64_t n, const int32_t *lut6,
                         int smooth, cudaStream_t s);
cudaError_t xk_nd_color_step(const uint8_t *st, int32_t *col, int64_t n, const int32_t *lut6,
                             int fade_in, int fade_out, int smooth, int plain, cudaStream_t s);

// RendererPlain over an int3 colour array of an N-D lattice
struct RenderGeo {
    int32_t ndim, a0, a1;
    int64_t size[XK_MAXDIM];
    int32_t smooth;             // 0: no SMOOTH_FACTOR division
};
// smallest and largest of `count` colour values into the device ints out[0],
// out[1] (render.cu)
cudaError_t xk_colors_minmax(const int32_t *col, int64_t count, int *out, cudaStream_t s);
bool xk_render_is_2d(const RenderGeo &g, int width, int height, int zoom);
cudaError_t xk_render_bits(const uint32_t *bits, void *img, bool bytes, const LifeGeo &lg, const int32_t *lut6,
                           int scale, const RenderGeo &g, int width, int height, int zoom, int dx, int dy,
                           cudaStream_t s);
cudaError_t xk_render_colors(const int32_t *col, int32_t *img, const RenderGeo &g, int width,
                             int height, int zoom, int dx, int dy, cudaStream_t s);
// the same frame as bytes (the int's low byte, as the reference's
// render() converts it)
cudaError_t xk_render_colors_u8(const int32_t *col, uint8_t *img, const RenderGeo &g, int width,
                                int height, int zoom, int dx, int dy, cudaStream_t s);

int xk_sm_count();

// generic interpreter (vm.cu)
struct VmGeo {
    int32_t ndim, nbr, torus, esz;
    int64_t n;
    int64_t size[XK_MAXDIM];
    int8_t delta[XK_MAXNBR][XK_MAXDIM];
    uint64_t border;             // static border: the whole off-board container
    int32_t color_kind, fade_in, fade_out, smooth;
};
cudaError_t xk_vm_run(const xk_vm_ins *code, int ncode, const uint64_t *consts,
                      const uint64_t *params, uint8_t *fld, int32_t *col, const VmGeo &g,
                      cudaStream_t s);

// Programs whose values fit 32 bits (vm_narrow.cu): the translation of a
// checked program (false: vm.cu runs it), and one pass of it.  Parameters are
// taken as 32-bit values: each used slot's image must be the sign (sign) or
// zero extension of its low half.  frame (a program that colours): also write
// the zoom-1 frame of a 2-D lattice.
struct XkVmParamUse {
    uint16_t slot;
    bool sign;
};
struct XkVmNarrow {
    std::vector<uint32_t> code, consts;
    std::vector<XkVmParamUse> params;
    int nloads = 0, nops = 0, nslots = 0, colors = 0;
    int threads = 0, smem = 0;   // of a block
};
bool xk_vm_translate(const xk_vm_ins *code, int ncode, const uint64_t *consts, int nregs, const VmGeo &g,
                     XkVmNarrow *out);
// whether it runs as a kernel argument (else from global memory)
inline bool xk_vm_narrow_is_argument(const XkVmNarrow &v) { return v.nops <= 1024 && v.consts.size() <= 512; }
cudaError_t xk_vm_run_narrow(const XkVmNarrow &v, const uint32_t *code, const uint32_t *consts,
                             const uint64_t *params, uint8_t *fld, int32_t *col, const VmGeo &g, cudaStream_t s,
                             uint8_t *frame = nullptr, int frame_smooth = 0);

// EvoLife family (evolife.cu)
cudaError_t xk_evolife_set_positional(const double *lut54);
// frame: null, or a W x H uint8 RGB frame written as RendererPlain renders the
// new colours at zoom 1 with no offset (frame_smooth: its SMOOTH_FACTOR, 0
// for none)
cudaError_t xk_evolife_step(const uint64_t *src, uint64_t *dst, int32_t *col, const xk_desc &d,
                            float mut_thresh, const int32_t *col_range, cudaStream_t s,
                            uint8_t *frame = nullptr, int frame_smooth = 0);

// Life with inherited colour channels (lifecolor.cu): 1 .. max generations,
// src -> dst, the colours updated, and (frames) each one's zoom-1 frame, one
// after another; color_range: smallest and largest colour that was loaded
int xk_lifecolor_max_generations();
cudaError_t xk_lifecolor_step(const uint32_t *src, uint32_t *dst, int32_t *col, const xk_desc &d, int generations,
                              const int32_t color_range[2], cudaStream_t s, uint8_t *frames = nullptr,
                              int frame_smooth = 0);

// per-cell noise (noise.cu): `generations` generations of every cell in one
// launch, in place; frames: null, or the zoom-1 frames of a 2-D lattice, one
// per generation, 3 n bytes each
cudaError_t xk_noise_step(uint16_t *cells, int32_t *col, const xk_desc &d, int64_t n, int generations,
                          cudaStream_t s, uint8_t *frames = nullptr, int frame_smooth = 0);
// one GraviCowboys generation, cells ping-pong (gravity.cu)
cudaError_t xk_gravity_step(const uint64_t *src, uint64_t *dst, int32_t *col, const xk_desc &d,
                            cudaStream_t s, uint8_t *frame, int frame_smooth);

// Programmatic dependent launch for kernels that run once per generation: the
// launch may begin while the previous kernel in the stream finishes, and the
// kernel calls xk_grid_dep_wait() before its first global-memory access
// (which returns once that kernel has completed and its writes are
// visible).  XK_PDL=0 in the environment launches plainly.
__device__ __forceinline__ void xk_grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

inline bool xk_pdl_enabled()
{
    const char *v = getenv("XK_PDL");
    return !(v && v[0] == '0');
}

template <typename... KArgs, typename... Args>
cudaError_t xk_launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                          Args... args)
{
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = xk_pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Bernoulli seeds (seed.cu): cells[off .. off + n) of a lattice =
// RandomState(seed).random_sample(n) < p, bit for bit
struct XkSeedJob {
    int64_t off, n;
    uint32_t seed, pad;
    double p;
};
cudaError_t xk_seed_bernoulli(const XkSeedJob *jobs, int count, uint8_t *cells, cudaStream_t s);

// mass-transfer family (mass.cu)
// Mass-transfer state on the device: rows of W cells at a pitch of W rounded
// up to a multiple of 4 (so a row starts on 16 bytes, as the tensor copies
// need); the padding cells hold 0.
inline int64_t xk_mass_pitch(int64_t W) { return (W + 3) / 4 * 4; }
// small: the lattice's total mass is below 2^30 (then every cell stays below
// it for good), which allows the fast-only kernel
// proj (only where xk_mass_fuses_projection()): also add the new state's
// column colour sums into proj (rows at the state's pitch, zero on entry; so
// wherever column sums are kept); with frame_prev, also
// write the zoom-1 frame of the previous generation from its sums proj_prev
// and zero proj_prev
cudaError_t xk_mass_step(const uint32_t *src, uint32_t *dst, unsigned long long *total,
                         const xk_desc &d, bool small, cudaStream_t s, uint32_t *proj = nullptr,
                         uint32_t *proj_prev = nullptr, uint8_t *frame_prev = nullptr);
// small: the total is below 2^30 (the kernel for it may allow more)
bool xk_mass_fuses_projection(const xk_desc &d, bool small);
// the kernel of lattices whose total is below 2^30 (mass_quads.cu): whether
// its indices span the lattice, whether it takes proj, one generation
bool xk_mass_quads_apply(const xk_desc &d);
bool xk_mass_quads_project(const xk_desc &d);
cudaError_t xk_mass_step_quads(const uint32_t *src, uint32_t *dst, unsigned long long *total, const xk_desc &d,
                               cudaStream_t s, uint32_t *proj, uint32_t *proj_prev, uint8_t *frame_prev);
// the W x H zoom-1 RendererPlain frame (axes (0, 1), no smoothing) from
// column colour sums
cudaError_t xk_mass_frame(const uint32_t *proj, uint8_t *frame, const xk_desc &d, cudaStream_t s);
// total of n cells into *out (64-bit)
cudaError_t xk_mass_sum(const uint32_t *src, int64_t n, unsigned long long *out, cudaStream_t s);
// true when a mass-transfer CTA gave up waiting for a tensor copy since the
// last call (the flag is cleared)
bool xk_mass_take_wait_failure();
// column colour sums over z; with `frame`, also the W x H RendererPlain frame
// over axes (0, 1) at zoom 1, no offset, as uint8 RGB
cudaError_t xk_mass_project(const uint32_t *src, uint32_t *proj, const xk_desc &d, cudaStream_t s,
                            uint8_t *frame = nullptr);
cudaError_t xk_mass_colors(const uint32_t *src, int32_t *col, const xk_desc &d, cudaStream_t s);
cudaError_t xk_mass_render(const uint32_t *proj, int32_t *img, const xk_desc &d, int width,
                           int height, int zoom, int dx, int dy, cudaStream_t s);
cudaError_t xk_mass_render_u8(const uint32_t *proj, uint8_t *img, const xk_desc &d, int width,
                              int height, int zoom, int dx, int dy, cudaStream_t s);
