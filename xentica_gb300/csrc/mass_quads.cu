// Mass-transfer generation of a lattice whose total mass is below 2^30 (then
// no cell ever reaches 2^30: mass is conserved and never negative, so no wall
// value is inside and m / 7 is one multiply-high; mass.cu has the model, the
// arithmetic and the general kernels).
//
//   m' = m - 6 q + sum of the six neighbours' q,     q = m / 7,
//
// where an off-board neighbour counts as the cell itself (it takes nothing and
// sends nothing), so nothing is counted per cell.
//
// A thread owns four consecutive cells (one 128-bit access) of R consecutive
// rows and marches along z with the planes before and after its own in
// registers; the next plane's rows are loaded one plane ahead.  Of 4 R cells
// it loads R + 2 rows (the rows above and below are its neighbours' own, so
// mostly L1 hits) and computes each row's q once; x neighbours beside the four
// cells come from the lanes beside (lanes 0 and 31 load one cell a row).  The
// quads of a plane are numbered row group by row group, so ragged widths
// waste no lanes.  No shared memory and no barrier in the loop.  The last row
// group is moved up to end at the last row; rows it shares are computed twice
// and counted once.
//
// Bound by the latency of its loads at 16 warps an SM, at 256^3 by DRAM.
// Microseconds a generation, against the general kernel's fast-only form
// (tensor copies into a shared ring, a barrier a plane, 163 instructions a warp
// and plane): 64^3 2.4 (3.4), 128^3 3.7 (5.5), 129 x 118 x 72 3.3 (5.5), 171 x
// 205 x 215 10.6 (16.9), 256^3 21.2 (24.5; 25.2 with every generation marching
// the same way); with a frame each 128^3 5.0 (7.5), 256^3 27.2 to 27.9 from
// run to run (29.9; 2 % more with the column sums in registers and the frame
// before the first planes' loads).
#include <string.h>

#include "xk_internal.cuh"

namespace {

struct QuadParams {
    int32_t W, H, D, P4;        // P4: quads of a (pitched) row
    int32_t groups, zc;         // row groups of a plane, planes of a run
    int32_t back;               // march towards lower z
    uint32_t quads;             // P4 * groups
};

__device__ __forceinline__ uint32_t q7(uint32_t m) { return __umulhi(m, 0x24924925u); }   // m / 7, m < 2^32 / 3

__device__ __forceinline__ uint4 q7(const uint4 &m) { return make_uint4(q7(m.x), q7(m.y), q7(m.z), q7(m.w)); }

__device__ __forceinline__ uint4 pick(bool a, const uint4 &x, const uint4 &y)
{
    return make_uint4(a ? x.x : y.x, a ? x.y : y.y, a ? x.z : y.z, a ? x.w : y.w);
}

__device__ __forceinline__ uint32_t colour(uint32_t m) { return min(m * 32u, 255u); }

__device__ __forceinline__ void add_shared(uint32_t at, uint32_t v)
{
    asm volatile("red.shared.add.u32 [%0], %1;" : : "r"(at), "r"(v) : "memory");
}

}  // namespace

// RAGGED: rows end inside a quad (W % 4 != 0); PROJ: also add the column
// colour sums of the written cells into proj, and with frame_prev write the
// previous generation's frame from proj_prev and zero it (as xk_k_mass_tma)
template <int R, bool RAGGED, bool PROJ>
__global__ void __launch_bounds__(128)
xk_k_mass_quads(const uint32_t *__restrict__ src, uint32_t *__restrict__ dst, unsigned long long *__restrict__ total,
                QuadParams p, uint32_t *__restrict__ proj, uint32_t *__restrict__ proj_prev,
                uint8_t *__restrict__ frame_prev)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = t < p.quads;
    const uint32_t tt = in ? t : p.quads - 1;
    const int yg = (int)(tt / (uint32_t)p.P4), xq = (int)(tt - (uint32_t)yg * (uint32_t)p.P4);
    const int lane = threadIdx.x & 31;
    const int y = min(yg * R, p.H - R), dup = yg * R - y;       // rows below dup belong to the group before
    const int z0 = blockIdx.y * p.zc, z1 = min(z0 + p.zc, p.D);
    const bool first = xq == 0, last = xq == p.P4 - 1;          // of their row
    const bool top = y == 0, bottom = y + R == p.H;
    const int end = (p.W - 1) & 3;                              // the last quad's last cell (RAGGED)
    const uint32_t pitch = (uint32_t)p.P4;
    const int64_t plane = (int64_t)p.P4 * p.H;                  // in quads
    const uint4 *cell = (const uint4 *)src + (int64_t)y * p.P4 + xq;
    // the rows above and below (their own first and last row where there is none)
    const int up = top ? 0 : -(int)pitch, down = (int)pitch * (bottom ? R - 1 : R);
    // the one cell beyond the warp that lanes 0 and 31 read
    const bool halo = lane == 0 ? !first : lane == 31 && !last;
    const int halo_at = lane == 0 ? -1 : 4;
    xk_grid_dep_wait();       // launched as a dependent of the previous generation
    // q of the plane before, cells and q of this one, its rows above and
    // below and halo cells as loaded
    uint4 qp[R], m[R], q[R], mu, md;
    uint32_t mh[R];
    {
        const int z = p.back ? z1 - 1 : z0;
        const uint4 *a = cell + (int64_t)z * plane;
#pragma unroll
        for (int r = 0; r < R; ++r) m[r] = __ldg(a + r * pitch);
        mu = __ldg(a + up);
        md = __ldg(a + down);
#pragma unroll
        for (int r = 0; r < R; ++r) mh[r] = halo ? __ldg((const uint32_t *)(a + r * pitch) + halo_at) : 0u;
        const uint4 *b = cell + (int64_t)(p.back ? min(z + 1, p.D - 1) : max(z - 1, 0)) * plane;
#pragma unroll
        for (int r = 0; r < R; ++r) qp[r] = __ldg(b + r * pitch);
    }
    if (PROJ && frame_prev) {
        // the previous generation's frame, four pixels a thread over the
        // whole grid, and its sums zeroed for the generation after this one
        // (here, while the first planes are on their way)
        const uint32_t quads = pitch * (uint32_t)p.H, threads = gridDim.x * gridDim.y * 128u;
        for (uint32_t i = blockIdx.y * gridDim.x * 128u + t; i < quads; i += threads) {
            const uint4 c = ((const uint4 *)proj_prev)[i];
            ((uint4 *)proj_prev)[i] = make_uint4(0u, 0u, 0u, 0u);
            const float D = (float)p.D;
            const uint32_t v[4] = {(uint32_t)(int)__fdiv_rn((float)c.x, D), (uint32_t)(int)__fdiv_rn((float)c.y, D),
                                   (uint32_t)(int)__fdiv_rn((float)c.z, D), (uint32_t)(int)__fdiv_rn((float)c.w, D)};
            const uint32_t row = i / pitch, x = 4u * (i - row * pitch);
            uint8_t *px = frame_prev + 3 * ((int64_t)row * p.W + x);
            if (!RAGGED && ((uintptr_t)frame_prev & 3u) == 0) {
                // r = g = b: bytes 0 0 0 1 | 1 1 2 2 | 2 3 3 3
                const uint32_t lo = __byte_perm(v[0], v[1], 0x0040), hi = __byte_perm(v[2], v[3], 0x0040);
                ((uint32_t *)px)[0] = __byte_perm(lo, 0, 0x1000);
                ((uint32_t *)px)[1] = __byte_perm(lo, hi, 0x4411);
                ((uint32_t *)px)[2] = __byte_perm(hi, 0, 0x1110);
            } else {
#pragma unroll
                for (int k = 0; k < 12; ++k)
                    if (x + k / 3 < (uint32_t)p.W) px[k] = (uint8_t)v[k / 3];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        qp[r] = q7(qp[r]);
        q[r] = q7(m[r]);
    }
    uint32_t sum = 0;                       // below 2^30: the whole lattice's total is
    // column sums, two 16-bit ones a word, in this thread's own words of
    // shared memory: added to without waiting, and no registers of the loop
    __shared__ uint32_t column[PROJ ? 2 * R : 1][128];
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(&column[0][threadIdx.x]);
    if (PROJ)
#pragma unroll
        for (int r = 0; r < 2 * R; ++r) column[PROJ ? r : 0][threadIdx.x] = 0u;
    for (int step = 0; step < z1 - z0; ++step) {
        const int z = p.back ? z1 - 1 - step : z0 + step;
        // the next plane (past the lattice: this one again, so that a cell's
        // missing neighbour is the cell itself)
        const uint4 *a = cell + (int64_t)(p.back ? max(z - 1, 0) : min(z + 1, p.D - 1)) * plane;
        uint4 mn[R];
#pragma unroll
        for (int r = 0; r < R; ++r) mn[r] = __ldg(a + r * pitch);
        const uint4 nu = __ldg(a + up), nd = __ldg(a + down);
        uint32_t nh[R];
#pragma unroll
        for (int r = 0; r < R; ++r) nh[r] = halo ? __ldg((const uint32_t *)(a + r * pitch) + halo_at) : 0u;
        const uint4 qu = q7(mu), qd = q7(md);
        uint4 *to = (uint4 *)dst + (int64_t)z * plane + (int64_t)y * p.P4 + xq;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint4 c = q[r], n = q7(mn[r]);
            const uint4 u = r > 0 ? q[r > 0 ? r - 1 : 0] : qu, d = r + 1 < R ? q[r + 1 < R ? r + 1 : r] : qd;
            const uint32_t qh = q7(mh[r]);
            uint32_t l = __shfl_up_sync(0xFFFFFFFFu, c.w, 1), x = __shfl_down_sync(0xFFFFFFFFu, c.x, 1);
            l = lane == 0 ? qh : l;
            x = lane == 31 ? qh : x;
            l = first ? c.x : l;
            x = last ? c.w : x;
            uint32_t r0 = c.y, r1 = c.z, r2 = c.w;
            if (RAGGED && last) {
                r0 = end == 0 ? c.x : r0;
                r1 = end == 1 ? c.y : r1;
                r2 = end == 2 ? c.z : r2;
            }
            uint4 o;
            o.x = m[r].x - 6u * c.x + l + r0 + u.x + d.x + qp[r].x + n.x;
            o.y = m[r].y - 6u * c.y + c.x + r1 + u.y + d.y + qp[r].y + n.y;
            o.z = m[r].z - 6u * c.z + c.y + r2 + u.z + d.z + qp[r].z + n.z;
            o.w = m[r].w - 6u * c.w + c.z + x + u.w + d.w + qp[r].w + n.w;
            if (RAGGED && last) {           // the row's padding stays 0
                o.y = end < 1 ? 0u : o.y;
                o.z = end < 2 ? 0u : o.z;
                o.w = end < 3 ? 0u : o.w;
            }
            if (in) to[r * pitch] = o;
            if (r >= dup) {
                sum += o.x + o.y + o.z + o.w;
                if (PROJ) {
                    add_shared(mine + 1024u * r, colour(o.x) + (colour(o.y) << 16));
                    add_shared(mine + 1024u * r + 512u, colour(o.z) + (colour(o.w) << 16));
                }
            }
            qp[r] = c;
            m[r] = mn[r];
            mh[r] = nh[r];
        }
#pragma unroll
        for (int r = 0; r < R; ++r) q[r] = q7(m[r]);
        mu = nu;
        md = nd;
    }
    if (PROJ && in) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (r < dup) continue;
            // two columns an atomic: a sum stays below 2^32, so none carries
            unsigned long long *pair = (unsigned long long *)(proj + 4 * ((int64_t)(y + r) * p.P4 + xq));
            const uint32_t a = column[2 * r][threadIdx.x], b = column[2 * r + 1][threadIdx.x];
            atomicAdd(pair, (unsigned long long)(a >> 16) << 32 | (a & 0xFFFFu));
            atomicAdd(pair + 1, (unsigned long long)(b >> 16) << 32 | (b & 0xFFFFu));
        }
    }
    // one atomic a block: they all hit one address
    __shared__ uint32_t sums[4];
    if (!in) sum = 0;
    sum = __reduce_add_sync(0xFFFFFFFFu, sum);
    if (lane == 0) sums[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(total, (unsigned long long)(sums[0] + sums[1] + sums[2] + sums[3]));
}

typedef void (*QuadKernel)(const uint32_t *, uint32_t *, unsigned long long *, QuadParams, uint32_t *, uint32_t *,
                           uint8_t *);

template <int R>
static QuadKernel quad_kernel(bool ragged, bool proj)
{
    if (ragged) return proj ? xk_k_mass_quads<R, true, true> : xk_k_mass_quads<R, true, false>;
    return proj ? xk_k_mass_quads<R, false, true> : xk_k_mass_quads<R, false, false>;
}

// Rows a thread and planes a run.  Without column sums: the pair that reads
// the fewest planes over its waves of resident blocks (4, 6 and 9 an SM by
// registers; a run reads two planes more than it writes, a thread of R rows
// R + 2; filling and draining the chip costs part of a run).  256^3: 4 rows and
// 14 planes 21.2 us a generation, 13 planes 24.5, 1 row 24.2.  With column sums
// one row a thread: a run ends in atomics for its columns (worth four planes
// more), and the more threads wait for them at once the better (128^3 5.0 against 6.7 us with 4 rows,
// 129 x 118 x 72 4.3 against 6.2, 256^3 27.0 against 27.4).
static void quad_shape(QuadParams &p, int &R, bool proj)
{
    const int64_t sms = xk_sm_count() > 0 ? xk_sm_count() : 1;
    const char *env = getenv("XK_MASS_ZC");
    const int forced = env ? atoi(env) : 0;
    // the generations of a run ask for the same shape again and again: a
    // search takes as long as a launch
    struct Found {
        int64_t sms;
        int32_t W, H, D;
        int forced, zc, R;
    };
    static thread_local Found last[2] = {};
    Found &f = last[proj ? 1 : 0];
    if (f.R && f.sms == sms && f.W == p.W && f.H == p.H && f.D == p.D && f.forced == forced) {
        p.zc = f.zc;
        R = f.R;
        return;
    }
    double best = 0;
    p.zc = 1;
    R = 0;
    for (int r : {4, 2, 1}) {
        if (p.H < r || (proj && r > 1)) continue;
        const int64_t blocks = ((int64_t)p.P4 * ((p.H + r - 1) / r) + 127) / 128;
        const int resident = r == 4 ? 4 : r == 2 ? 6 : 9;
        for (int zc = 1; zc <= 256 && zc <= p.D; ++zc) {
            const int z = forced > 0 ? forced : zc;
            const int64_t runs = (p.D + z - 1) / z;
            const int64_t waves = (blocks * runs + sms * resident - 1) / (sms * resident);
            const double cost = ((double)waves + (proj ? 0.5 : 0.25)) * (z + (proj ? 6 : 2)) * (r + 2) * resident;
            if (!R || cost < best) {
                best = cost;
                p.zc = z;
                R = r;
            }
        }
    }
    f = Found{sms, p.W, p.H, p.D, forced, p.zc, R};
}

static QuadParams quad_params(const xk_desc &d, int &R, bool proj)
{
    QuadParams p;
    p.W = (int32_t)d.size[0];
    p.H = (int32_t)d.size[1];
    p.D = (int32_t)d.size[2];
    p.P4 = (int32_t)(xk_mass_pitch(p.W) / 4);
    quad_shape(p, R, proj);
    p.back = 0;
    p.groups = (p.H + R - 1) / R;
    p.quads = (uint32_t)p.P4 * (uint32_t)p.groups;
    return p;
}

bool xk_mass_quads_apply(const xk_desc &d)
{
    // 32-bit quad numbers and grids
    return (int64_t)xk_mass_pitch(d.size[0]) * d.size[1] <= (1ll << 31) && d.size[2] <= 65535 &&
           d.size[0] * d.size[1] < (1ll << 31);
}

bool xk_mass_quads_project(const xk_desc &d)
{
    int R = 0;
    return quad_params(d, R, true).zc <= 256;      // the 16-bit column sums of a run of planes
}

cudaError_t xk_mass_step_quads(const uint32_t *src, uint32_t *dst, unsigned long long *total, const xk_desc &d,
                               cudaStream_t s, uint32_t *proj, uint32_t *proj_prev, uint8_t *frame_prev)
{
    int R = 0;
    QuadParams p = quad_params(d, R, proj != nullptr);
    if (proj && p.zc > 256) return cudaErrorNotSupported;
    // The two buffers of a lattice larger than half of L2 do not stay there
    // whole: generations march in alternate directions, so that each starts on
    // the planes the one before wrote last.
    p.back = src < dst;
    const bool ragged = p.W % 4 != 0;
    const QuadKernel k = R == 4 ? quad_kernel<4>(ragged, proj != nullptr)
                         : R == 2 ? quad_kernel<2>(ragged, proj != nullptr) : quad_kernel<1>(ragged, proj != nullptr);
    const dim3 grid((p.quads + 127) / 128, (unsigned)((p.D + p.zc - 1) / p.zc));
    return xk_launch_pdl(k, grid, dim3(128), 0, s, src, dst, total, p, proj, proj_prev, frame_prev);
}
