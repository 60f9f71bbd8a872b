// The interpreter for programs whose values fit 32 bits (vm.cu runs the rest).
//
// The host translates a checked program (xk_vm_translate) into operations on
// 32-bit values: conversions and moves that leave a value's low half alone
// only rename it and constants become operands.  What
// vm.cu computes on 64-bit images is the same in the low halves as long as
// the translation knows every image to be the sign or the zero extension of
// its low half where an operation looks at more than that; where it does not
// know, the program stays with vm.cu.
//
// A thread runs four cells, 32 apart: a register is 16 bytes of shared memory
// (a slot of its warp, lane after lane, so no bank conflicts), one dispatch
// serves four cells, loads before the first store are issued together.
// Neighbour cells are found from per-thread tables of each axis' three
// offsets.  Programs of up to 1024 operations are kernel arguments.  An
// operation's dispatch covers the next one's operand loads; an operand that
// is its result is taken from registers.
//
// An operation whose result only the next one reads is joined with it (63
// pairs of the common integer operations, and the addition of a comparison of
// a masked value), stores of one value to several planes are one.
//
// Bound by the latency of an operation (fetch, dispatch, shared memory: about
// 240 cycles a warp, 360 of a pair, the same at three warps a scheduler as at
// one).  640 x 360 cells, 65 absorb operations (123 as loaded) and 11 of emit
// before the joins, a frame a generation: 16.0 us, 18.3 without them, against
// 81.6 us with vm.cu's 64-bit registers in local memory and one cell a thread.
// Measured and not kept: eight cells a thread (16.8 against 16.7 us on such a
// program, 108 against 107 at 1920 x 1080), the code in shared memory (17.8),
// operand loads behind the dispatch (19.9), the third operand loaded ahead as
// the others are (16.9 against 16.7 before stores were joined).
#include <string.h>

#include <algorithm>
#include <vector>

#include "xk_internal.cuh"

#include "frame.cuh"

enum {
    N_ADD, N_SUB, N_MUL, N_AND, N_OR, N_XOR, N_SHL, N_SHRS, N_SHRU, N_DIVS, N_DIVU, N_MODS, N_MODU,
    N_LTS, N_LTU, N_LES, N_LEU, N_EQ, N_NE,
    N_FADD, N_FSUB, N_FMUL, N_FDIV, N_FLT, N_FLE, N_FEQ, N_FNE,
    N_NEG, N_NOT, N_ABSS, N_FNEG, N_FABS, N_SEL, N_BOOL, N_I2F, N_U2F, N_F2S, N_F2U, N_F2B, N_POPC, N_MOV,
    N_PARAM, N_LOAD, N_STORE, N_COLOR,
    N_STORES,                   // one value to several planes (imm: their mask), as emit copies a cell
    N_COUNT,                    // ((a & b) == c) + d: one more neighbour in a state
    N_PAIR                      // two operations in one: N_PAIR + first * VN_SECONDS + second
};
// An operation whose result only the next one reads joins it: (a first b)
// second c, for these (second's operands swapped where it commutes)
constexpr int VN_FIRST[] = {N_ADD, N_MUL, N_AND, N_OR, N_SHRU, N_SHL, N_EQ, N_LTU, N_LTS};
constexpr int VN_SECOND[] = {N_ADD, N_MUL, N_AND, N_OR, N_EQ, N_SHRU, N_SHL};
constexpr int VN_SECONDS = 7;
enum { NF_A = 1, NF_B = 2, NF_C = 4, NF_STORE = 8, NF_D = 16 };   // operands and result an operation has
#define XK_VN_CONST 0x8000     // a slot number with this bit is a constant's

// translation: loads: a = kind (0 own cell, 1 neighbour), c = plane, imm = the
// neighbour's offsets + 1, two bits an axis; stores: imm = plane; parameters:
// a = slot; a fourth operand: imm.
struct XkVnOp {
    uint16_t op, flags, dst, a, b, c;
    uint32_t imm;
};

// What the kernel reads.  Loads: c = kind (0 own cell, 1 neighbour), imm as
// above; stores and loads: plane (elsewhere a fourth operand); parameters: c =
// slot.
struct XkVnCode {
    uint16_t dst, a, b, c, op, plane;
    uint32_t imm;
};
static_assert(sizeof(XkVnCode) == 16, "an operation is one 16-byte load");

// A program as a kernel argument: read through the constant bank, so the
// compiler sees that operations and places are the same for the whole warp
// and keeps them, and the dispatch, on the uniform path.  CODE = 0: a program
// too long for that, in global memory.
template <int CODE, int CONSTS>
struct VnProgram {
    alignas(16) XkVnCode code[CODE + 2];
    uint32_t consts[CONSTS];
};

template <>
struct VnProgram<0, 0> {
    const XkVnCode *code;
    const uint32_t *consts;
};

struct VnParams {
    const uint64_t *params;
    int32_t nloads, nops, nconsts, nslots, colors;    // nslots with the constants'
    uint8_t *frame;              // null, or the zoom-1 RendererPlain frame of a 2-D lattice
    int32_t frame_smooth;
    int32_t ndim, torus;
    uint32_t n, border;
    uint32_t size[XK_MAXDIM];
    int32_t color_kind, fade_in, neg_fade_out, smooth;
};

#define XK_VN_OFF 0x80000000u    // an off-board axis offset (sums of on-board ones stay below)

template <int ESZ>
__device__ __forceinline__ uint32_t vn_ld(const uint8_t *p, uint32_t i)
{
    return ESZ == 4 ? ((const uint32_t *)p)[i] : ESZ == 2 ? ((const uint16_t *)p)[i] : p[i];
}

template <int ESZ>
__device__ __forceinline__ void vn_st(uint8_t *p, uint32_t i, uint32_t v)
{
    if (ESZ == 4) ((uint32_t *)p)[i] = v;
    else if (ESZ == 2) ((uint16_t *)p)[i] = (uint16_t)v;
    else p[i] = (uint8_t)v;
}

// C's float -> unsigned / int as vm.cu converts: NaN 0, truncation, negative
// 0 for unsigned, the low 32 bits of the 64-bit result
__device__ __forceinline__ uint32_t vn_f2u(float f)
{
    return f > 0.0f ? (uint32_t)(unsigned long long)__float2ll_rz(f) : 0u;
}

__device__ __forceinline__ uint32_t vn_f2s(float f)
{
    return f == f ? (uint32_t)(unsigned long long)__float2ll_rz(f) : 0u;
}

__device__ __forceinline__ uint32_t vn_divs(uint32_t x, uint32_t y, bool mod)
{
    const int32_t a = (int32_t)x, b = (int32_t)y;
    if (b == 0) return 0;
    if (b == -1) return mod ? 0u : 0u - x;
    return (uint32_t)(mod ? a % b : a / b);
}

// shared memory by 32-bit address
__device__ __forceinline__ uint4 vn_lds(uint32_t at)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
    return v;
}

__device__ __forceinline__ void vn_sts(uint32_t at, const uint4 &v)
{
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" : : "r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}

template <int OP>
__device__ __forceinline__ uint32_t vn_do(uint32_t x, uint32_t y)
{
    return OP == N_ADD ? x + y : OP == N_MUL ? x * y : OP == N_AND ? x & y : OP == N_OR ? x | y
           : OP == N_SHRU ? x >> (y & 31u) : OP == N_SHL ? x << (y & 31u) : OP == N_EQ ? (uint32_t)(x == y)
           : OP == N_LTU ? (uint32_t)(x < y) : (uint32_t)((int32_t)x < (int32_t)y);
}

template <int FIRST, int SECOND>
__device__ __forceinline__ uint4 vn_pair(const uint4 &a, const uint4 &b, const uint4 &c)
{
    constexpr int F = VN_FIRST[FIRST], S = VN_SECOND[SECOND];
    return make_uint4(vn_do<S>(vn_do<F>(a.x, b.x), c.x), vn_do<S>(vn_do<F>(a.y, b.y), c.y),
                      vn_do<S>(vn_do<F>(a.z, b.z), c.z), vn_do<S>(vn_do<F>(a.w, b.w), c.w));
}

#define XK_VN_PAIR(F, S)                                                                                     \
    case N_PAIR + (F) * VN_SECONDS + (S): acc = vn_pair<F, S>(va, vb, get(o.y >> 16)); break;
#define XK_VN_PAIRS(F)                                                                                       \
    XK_VN_PAIR(F, 0) XK_VN_PAIR(F, 1) XK_VN_PAIR(F, 2) XK_VN_PAIR(F, 3) XK_VN_PAIR(F, 4) XK_VN_PAIR(F, 5)    \
    XK_VN_PAIR(F, 6)

#define XK_VN_ONE(f, expr)                                                                                   \
    {                                                                                                        \
        const uint32_t x = va.f, y = vb.f;                                                                   \
        (void)y;                                                                                             \
        acc.f = (uint32_t)(expr);                                                                            \
    }
#define XK_VN_EACH(expr)                                                                                     \
    {                                                                                                        \
        XK_VN_ONE(x, expr) XK_VN_ONE(y, expr) XK_VN_ONE(z, expr) XK_VN_ONE(w, expr)                          \
        break;                                                                                               \
    }
#define XK_VN_F(v) __uint_as_float(v)

// one pass of a program
template <int ESZ, class PROG>
__global__ void __launch_bounds__(128)
xk_k_vm_narrow(uint8_t *__restrict__ fld, int32_t *__restrict__ col, const __grid_constant__ VnParams p,
               const __grid_constant__ PROG prog)
{
    // [warp][slots, the constants', 3 ndim table rows][lane]: 16 bytes, a
    // thread's four cells (32 apart: a warp's 128 are consecutive)
    extern __shared__ uint4 vn_sm[];
    constexpr uint32_t SLOT = 512u;
    constexpr int C = 4;
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(vn_sm) +
                          (tid >> 5) * (uint32_t)(p.nslots + 3 * p.ndim) * SLOT + lane * 16u;
    const uint32_t tab = mine + (uint32_t)p.nslots * SLOT;
    const uint32_t w0 = (uint32_t)C * (blockIdx.x * blockDim.x + (tid & ~31u));   // the warp's first cell
    if (w0 >= p.n) return;                 // whole warps; no block-wide synchronisation below
    auto put = [&](uint32_t slot, const uint4 &v) { vn_sts(mine + slot * SLOT, v); };
    auto get = [&](uint32_t slot) { return vn_lds(mine + slot * SLOT); };
    for (int k = 0; k < p.nconsts; ++k) {
        const uint32_t c = prog.consts[k];
        put((uint32_t)(p.nslots - p.nconsts + k), make_uint4(c, c, c, c));
    }
    uint32_t cell[C];
#pragma unroll
    for (int k = 0; k < C; ++k) cell[k] = min(w0 + 32u * k + lane, p.n - 1u);
    {
        // each axis: what its -1, 0, +1 neighbour adds to a flat index
        uint32_t rest[C], stride = 1;
#pragma unroll
        for (int k = 0; k < C; ++k) rest[k] = cell[k];
        for (int d = 0; d < p.ndim; ++d) {
            const uint32_t size = p.size[d];
            uint32_t t[3][C];
#pragma unroll
            for (int k = 0; k < C; ++k) {
                const uint32_t q = d + 1 < p.ndim ? rest[k] / size : 0u, x = rest[k] - q * size;
                rest[k] = q;
                t[1][k] = x * stride;
                t[0][k] = x > 0 ? (x - 1) * stride : p.torus ? (size - 1) * stride : XK_VN_OFF;
                t[2][k] = x + 1 < size ? (x + 1) * stride : p.torus ? 0u : XK_VN_OFF;
            }
#pragma unroll
            for (int o = 0; o < 3; ++o)
                vn_sts(tab + (uint32_t)(3 * d + o) * SLOT, make_uint4(t[o][0], t[o][1], t[o][2], t[o][3]));
            stride *= size;
        }
    }
    xk_grid_dep_wait();                    // launched as a dependent of the pass before
    auto op_at = [&](int at) { return *(const uint4 *)&prog.code[at]; };
    // a load: kind, plane, offsets
    auto load = [&](uint32_t kind, uint32_t which, uint32_t imm) {
        const uint8_t *plane = fld + (int64_t)p.n * which * ESZ;
        uint4 v;
        if (kind == 0) {
            v.x = vn_ld<ESZ>(plane, cell[0]);
            v.y = vn_ld<ESZ>(plane, cell[1]);
            v.z = vn_ld<ESZ>(plane, cell[2]);
            v.w = vn_ld<ESZ>(plane, cell[3]);
            return v;
        }
        uint4 j = make_uint4(0, 0, 0, 0), f = j;
        for (int d = 0; d < p.ndim; ++d) {
            const uint4 t = vn_lds(tab + (3u * d + ((imm >> (2 * d)) & 3u)) * SLOT);
            j.x += t.x;
            j.y += t.y;
            j.z += t.z;
            j.w += t.w;
            f.x |= t.x;
            f.y |= t.y;
            f.z |= t.z;
            f.w |= t.w;
        }
        if (p.torus) {
            v.x = vn_ld<ESZ>(plane, j.x);
            v.y = vn_ld<ESZ>(plane, j.y);
            v.z = vn_ld<ESZ>(plane, j.z);
            v.w = vn_ld<ESZ>(plane, j.w);
        } else {
            v.x = f.x & XK_VN_OFF ? p.border : vn_ld<ESZ>(plane, j.x);
            v.y = f.y & XK_VN_OFF ? p.border : vn_ld<ESZ>(plane, j.y);
            v.z = f.z & XK_VN_OFF ? p.border : vn_ld<ESZ>(plane, j.z);
            v.w = f.w & XK_VN_OFF ? p.border : vn_ld<ESZ>(plane, j.w);
        }
        return v;
    };
    // the program's leading loads, four in flight at a time
    int pc = 0;
    for (; pc + 4 <= p.nloads; pc += 4) {
        uint4 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const XkVnCode &o = prog.code[pc + q];
            v[q] = load(o.c, o.plane, o.imm);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) put(prog.code[pc + q].dst, v[q]);
    }
    for (; pc < p.nloads; ++pc) {
        const XkVnCode &o = prog.code[pc];
        put(o.dst, load(o.c, o.plane, o.imm));
    }
    // the colours faded from, while the program runs
    int old[3 * C];
    const bool fades = p.colors && p.color_kind == XK_COLOR_MOVING_AVERAGE;
#pragma unroll
    for (int k = 0; k < 3 * C; ++k) old[k] = fades ? col[3 * (int64_t)cell[k / 3] + k % 3] : 0;
    // One operation's dispatch covers the next one's operand loads: an
    // operand that is this operation's result is taken from it instead.
    uint4 o = op_at(pc), nx = op_at(pc + 1);     // one past the last operation is readable
    uint4 va = get(o.x >> 16), vb = get(o.y & 0xFFFFu);
    for (; pc < p.nops; ++pc) {
        const uint4 nn = op_at(pc + 2);          // two past it too
        const uint32_t dst = o.x & 0xFFFFu, na = nx.x >> 16, nb = nx.y & 0xFFFFu;
        const uint4 pa = get(na), pb = get(nb);
        uint4 acc = va;
        switch (o.z & 0xFFFFu) {
        case N_ADD: XK_VN_EACH(x + y)
        case N_SUB: XK_VN_EACH(x - y)
        case N_MUL: XK_VN_EACH(x * y)
        case N_AND: XK_VN_EACH(x & y)
        case N_OR: XK_VN_EACH(x | y)
        case N_XOR: XK_VN_EACH(x ^ y)
        case N_SHL: XK_VN_EACH(x << (y & 31u))
        case N_SHRS: XK_VN_EACH((int32_t)x >> (y & 31u))
        case N_SHRU: XK_VN_EACH(x >> (y & 31u))
        case N_DIVS: XK_VN_EACH(vn_divs(x, y, false))
        case N_DIVU: XK_VN_EACH(y ? x / y : 0u)
        case N_MODS: XK_VN_EACH(vn_divs(x, y, true))
        case N_MODU: XK_VN_EACH(y ? x % y : 0u)
        case N_LTS: XK_VN_EACH((int32_t)x < (int32_t)y)
        case N_LTU: XK_VN_EACH(x < y)
        case N_LES: XK_VN_EACH((int32_t)x <= (int32_t)y)
        case N_LEU: XK_VN_EACH(x <= y)
        case N_EQ: XK_VN_EACH(x == y)
        case N_NE: XK_VN_EACH(x != y)
        case N_FADD: XK_VN_EACH(__float_as_uint(__fadd_rn(XK_VN_F(x), XK_VN_F(y))))
        case N_FSUB: XK_VN_EACH(__float_as_uint(__fsub_rn(XK_VN_F(x), XK_VN_F(y))))
        case N_FMUL: XK_VN_EACH(__float_as_uint(__fmul_rn(XK_VN_F(x), XK_VN_F(y))))
        case N_FDIV: XK_VN_EACH(__float_as_uint(__fdiv_rn(XK_VN_F(x), XK_VN_F(y))))
        case N_FLT: XK_VN_EACH(XK_VN_F(x) < XK_VN_F(y))
        case N_FLE: XK_VN_EACH(XK_VN_F(x) <= XK_VN_F(y))
        case N_FEQ: XK_VN_EACH(XK_VN_F(x) == XK_VN_F(y))
        case N_FNE: XK_VN_EACH(XK_VN_F(x) != XK_VN_F(y))
        case N_NEG: XK_VN_EACH(0u - x)
        case N_NOT: XK_VN_EACH(~x)
        case N_ABSS: XK_VN_EACH((int32_t)x < 0 ? 0u - x : x)
        case N_FNEG: XK_VN_EACH(__float_as_uint(-XK_VN_F(x)))
        case N_FABS: XK_VN_EACH(__float_as_uint(fabsf(XK_VN_F(x))))
        case N_SEL: {
            const uint4 vc = get(o.y >> 16);
            acc = make_uint4(va.x ? vb.x : vc.x, va.y ? vb.y : vc.y, va.z ? vb.z : vc.z, va.w ? vb.w : vc.w);
            break;
        }
        case N_BOOL: XK_VN_EACH(x != 0)
        case N_I2F: XK_VN_EACH(__float_as_uint(__int2float_rn((int32_t)x)))
        case N_U2F: XK_VN_EACH(__float_as_uint(__uint2float_rn(x)))
        case N_F2S: XK_VN_EACH(vn_f2s(XK_VN_F(x)))
        case N_F2U: XK_VN_EACH(vn_f2u(XK_VN_F(x)))
        case N_F2B: XK_VN_EACH(fabsf(XK_VN_F(x)) >= 1.0f)
        case N_POPC: XK_VN_EACH(__popc(x))
        case N_MOV: XK_VN_EACH(x)
        case N_PARAM: {
            const uint32_t v = (uint32_t)__ldg(p.params + (o.y >> 16));
            acc = make_uint4(v, v, v, v);
            break;
        }
        case N_LOAD: {
            acc = load(o.y >> 16, o.z >> 16, o.w);
            break;
        }
        case N_STORE: {
            uint8_t *plane = fld + (int64_t)p.n * (o.z >> 16) * ESZ;
            const uint32_t v[4] = {va.x, va.y, va.z, va.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t i = w0 + 32u * k + lane;
                if (i < p.n) vn_st<ESZ>(plane, i, v[k]);
            }
            break;
        }
        case N_COLOR: {
            const uint4 vc = get(o.y >> 16);
            const uint32_t r[4] = {va.x, va.y, va.z, va.w}, g[4] = {vb.x, vb.y, vb.z, vb.w};
            const uint32_t b[4] = {vc.x, vc.y, vc.z, vc.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t i = w0 + 32u * k + lane;
                int c[3] = {(int)r[k], (int)g[k], (int)b[k]};
                if (fades) {
                    // a second colour of the program fades from this one
#pragma unroll
                    for (int ch = 0; ch < 3; ++ch)
                        old[3 * k + ch] = c[ch] = xk_fade((int)((uint32_t)c[ch] * (uint32_t)p.smooth),
                                                          old[3 * k + ch], p.fade_in, p.neg_fade_out);
                }
                if (i >= p.n) continue;
                int32_t *to = col + 3 * (int64_t)i;
                to[0] = c[0];
                to[1] = c[1];
                to[2] = c[2];
                if (!p.frame) continue;
                uint8_t *px = p.frame + 3 * (int64_t)i;
                if (p.frame_smooth <= 1 && xk_px_small(c[0]) && xk_px_small(c[1]) && xk_px_small(c[2])) {
                    px[0] = (uint8_t)c[0];
                    px[1] = (uint8_t)c[1];
                    px[2] = (uint8_t)c[2];
                } else {
                    px[0] = (uint8_t)xk_pixel(c[0], p.frame_smooth);
                    px[1] = (uint8_t)xk_pixel(c[1], p.frame_smooth);
                    px[2] = (uint8_t)xk_pixel(c[2], p.frame_smooth);
                }
            }
            break;
        }
        case N_STORES: {
            const uint32_t v[4] = {va.x, va.y, va.z, va.w};
            for (uint32_t left = o.w; left != 0; left &= left - 1) {
                uint8_t *plane = fld + (int64_t)p.n * (__ffs((int)left) - 1) * ESZ;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t i = w0 + 32u * k + lane;
                    if (i < p.n) vn_st<ESZ>(plane, i, v[k]);
                }
            }
            break;
        }
        case N_COUNT: {
            const uint4 vc = get(o.y >> 16), vd = get(o.z >> 16);
            acc = make_uint4(((va.x & vb.x) == vc.x) + vd.x, ((va.y & vb.y) == vc.y) + vd.y,
                             ((va.z & vb.z) == vc.z) + vd.z, ((va.w & vb.w) == vc.w) + vd.w);
            break;
        }
        XK_VN_PAIRS(0)
        XK_VN_PAIRS(1)
        XK_VN_PAIRS(2)
        XK_VN_PAIRS(3)
        XK_VN_PAIRS(4)
        XK_VN_PAIRS(5)
        XK_VN_PAIRS(6)
        XK_VN_PAIRS(7)
        XK_VN_PAIRS(8)
        default: break;
        }
        put(dst, acc);                           // operations without a result have a slot nothing reads
        va = na == dst ? acc : pa;
        vb = nb == dst ? acc : pb;
        o = nx;
        nx = nn;
    }
}

// ---------------------------------------------------------------------------
// translation

namespace {

// what is known of a register's value: its slot (a physical register's, or a
// constant's), how its 64-bit image extends the low half, and an upper bound
enum Ext { BOTH, SIGN, ZERO };      // BOTH: below 2^31, so the same either way
struct Known {
    int slot = -1;
    Ext ext = BOTH;
    uint32_t hi = 0;
};

enum { T_BOOL, T_U8, T_U16, T_I32, T_U32, T_I64, T_U64, T_F32, T_F64 };

Known bounded(uint64_t hi, int ty)
{
    Known k;
    if (hi < (1ull << 31)) {
        k.hi = (uint32_t)hi;
        return k;
    }
    k.ext = ty == T_I32 ? SIGN : ZERO;
    k.hi = 0xFFFFFFFFu;
    return k;
}

uint64_t ones(uint64_t hi)          // the smallest 2^b - 1 not below hi
{
    uint64_t m = 0;
    while (m < hi) m = 2 * m + 1;
    return m;
}

struct Translator {
    const uint64_t *consts;
    const VmGeo &g;
    std::vector<XkVnOp> ops;
    std::vector<uint32_t> pool;
    std::vector<Known> reg;
    std::vector<XkVmParamUse> params;
    int nregs;
    bool ok = true;

    Translator(const uint64_t *c, int nr, const VmGeo &geo) : consts(c), g(geo), reg(nr), nregs(nr)
    {
        for (int r = 0; r < nr; ++r) reg[r].slot = constant(0);     // read before written: 0
    }

    int constant(uint32_t v)
    {
        for (size_t k = 0; k < pool.size(); ++k)
            if (pool[k] == v) return XK_VN_CONST | (int)k;
        pool.push_back(v);
        return XK_VN_CONST | (int)(pool.size() - 1);
    }

    void emit(int op, int dst, int a = -1, int b = -1, int c = -1, uint32_t imm = 0)
    {
        XkVnOp o;
        memset(&o, 0, sizeof(o));
        o.op = (uint16_t)op;
        if (dst >= 0) {
            o.dst = (uint16_t)dst;
            o.flags |= NF_STORE;
        }
        if (a >= 0) {
            o.a = (uint16_t)a;
            o.flags |= NF_A;
        }
        if (b >= 0) {
            o.b = (uint16_t)b;
            o.flags |= NF_B;
        }
        if (c >= 0) {
            o.c = (uint16_t)c;
            o.flags |= NF_C;
        }
        o.imm = imm;
        ops.push_back(o);
    }

    // register r's own slot is about to be written: registers that merely
    // name it get a copy first
    void claim(int r)
    {
        int copy = -1;
        for (int q = 0; q < nregs; ++q)
            if (q != r && reg[q].slot == r) {
                if (copy < 0) {
                    emit(N_MOV, q, r);
                    copy = q;
                }
                reg[q].slot = copy;
            }
    }

    void result(int r, const Known &k, int op, int a = -1, int b = -1, int c = -1, uint32_t imm = 0)
    {
        claim(r);
        // operands that named r's old value still read it: the write comes last
        emit(op, r, a, b, c, imm);
        reg[r] = k;
        reg[r].slot = r;
    }

    void alias(int r, Known k)
    {
        if (k.slot != r) claim(r);
        // claim may have moved what k names
        reg[r] = k;
    }

    bool known_const(const Known &k, uint32_t &v) const
    {
        if (!(k.slot & XK_VN_CONST)) return false;
        v = pool[k.slot & (XK_VN_CONST - 1)];
        return true;
    }

    void binary(const xk_vm_ins &in);
    void convert(const xk_vm_ins &in);
    void one(const xk_vm_ins &in);
};

void Translator::binary(const xk_vm_ins &in)
{
    const int ty = in.ty, op = in.op;
    const Known a = reg[in.a], b = reg[in.b];
    if (ty == T_F32) {
        static const int fop[] = {N_FADD, N_FSUB, N_FMUL, N_FDIV};
        Known f;
        f.ext = ZERO;
        f.hi = 0xFFFFFFFFu;
        if (op >= 10 && op <= 13) return result(in.dst, f, fop[op - 10], a.slot, b.slot);
        if (op < 20) return alias(in.dst, Known{constant(0), BOTH, 0});      // as vm.cu: 0
        switch (op) {
        case 20: return result(in.dst, bounded(1, ty), N_FLT, a.slot, b.slot);
        case 21: return result(in.dst, bounded(1, ty), N_FLE, a.slot, b.slot);
        case 22: return result(in.dst, bounded(1, ty), N_FLT, b.slot, a.slot);
        case 23: return result(in.dst, bounded(1, ty), N_FLE, b.slot, a.slot);
        case 24: return result(in.dst, bounded(1, ty), N_FEQ, a.slot, b.slot);
        default: return result(in.dst, bounded(1, ty), N_FNE, a.slot, b.slot);
        }
    }
    if (ty != T_I32 && ty != T_U32) return alias(in.dst, Known{constant(0), BOTH, 0});   // as vm.cu: 0
    const bool s = ty == T_I32, small = a.ext == BOTH && b.ext == BOTH;
    uint32_t cv = 0;
    const bool bc = known_const(b, cv);
    auto any = [&]() { return bounded(0xFFFFFFFFull, ty); };
    switch (op) {
    case 10: return result(in.dst, small ? bounded((uint64_t)a.hi + b.hi, ty) : any(), N_ADD, a.slot, b.slot);
    case 11: return result(in.dst, any(), N_SUB, a.slot, b.slot);
    case 12: {
        const uint64_t m = (uint64_t)a.hi * b.hi;
        return result(in.dst, small && m < (1ull << 31) ? bounded(m, ty) : any(), N_MUL, a.slot, b.slot);
    }
    case 13:
        return result(in.dst, small || (!s && a.ext != SIGN) ? bounded(a.hi, ty) : any(), s && !small ? N_DIVS : N_DIVU,
                      a.slot, b.slot);
    case 14:
        return result(in.dst, bc && cv && (!s || small) ? bounded(cv - 1, ty) : small ? bounded(a.hi, ty) : any(),
                      s && !small ? N_MODS : N_MODU, a.slot, b.slot);
    case 15:
        return result(in.dst,
                      a.ext == BOTH && b.ext == BOTH ? bounded(std::min(a.hi, b.hi), ty)
                      : a.ext == BOTH ? bounded(a.hi, ty) : b.ext == BOTH ? bounded(b.hi, ty) : any(),
                      N_AND, a.slot, b.slot);
    case 16:
        return result(in.dst, small ? bounded(ones(std::max(a.hi, b.hi)), ty) : any(), N_OR, a.slot, b.slot);
    case 17:
        return result(in.dst, small ? bounded(ones(std::max(a.hi, b.hi)), ty) : any(), N_XOR, a.slot, b.slot);
    case 18: {
        const uint64_t m = bc ? (uint64_t)a.hi << (cv & 31u) : 1ull << 40;
        return result(in.dst, a.ext == BOTH && m < (1ull << 31) ? bounded(m, ty) : any(), N_SHL, a.slot, b.slot);
    }
    case 19: {
        const bool plain = !s || a.ext == BOTH;                // shifts in zeros
        Known k = any();
        if (a.ext == BOTH) k = bounded(a.hi >> (bc ? cv & 31u : 0u), ty);
        else if (!s && bc) k = bounded(0xFFFFFFFFu >> (cv & 31u), ty);
        return result(in.dst, k, plain ? N_SHRU : N_SHRS, a.slot, b.slot);
    }
    case 20: return result(in.dst, bounded(1, ty), s ? N_LTS : N_LTU, a.slot, b.slot);
    case 21: return result(in.dst, bounded(1, ty), s ? N_LES : N_LEU, a.slot, b.slot);
    case 22: return result(in.dst, bounded(1, ty), s ? N_LTS : N_LTU, b.slot, a.slot);
    case 23: return result(in.dst, bounded(1, ty), s ? N_LES : N_LEU, b.slot, a.slot);
    case 24: return result(in.dst, bounded(1, ty), N_EQ, a.slot, b.slot);
    default: return result(in.dst, bounded(1, ty), N_NE, a.slot, b.slot);
    }
}

void Translator::convert(const xk_vm_ins &in)
{
    const int from = in.b, to = in.ty;
    const Known a = reg[in.a];
    if (from == to) return alias(in.dst, a);
    auto mask = [&](uint32_t m, int slot, const Known &k) {
        if (k.ext == BOTH && k.hi <= m) return alias(in.dst, k);
        return result(in.dst, bounded(m, to), N_AND, slot, constant(m));
    };
    if (from == T_F32) {
        if (to == T_BOOL) return result(in.dst, bounded(1, to), N_F2B, a.slot);
        if (to == T_I32) return result(in.dst, bounded(0xFFFFFFFFu, T_I32), N_F2S, a.slot);
        result(in.dst, bounded(0xFFFFFFFFu, T_U32), N_F2U, a.slot);
        if (to == T_U8) return mask(0xFFu, in.dst, reg[in.dst]);
        if (to == T_U16) return mask(0xFFFFu, in.dst, reg[in.dst]);
        return;
    }
    if (to == T_F32) {
        Known f;
        f.ext = ZERO;
        f.hi = 0xFFFFFFFFu;
        return result(in.dst, f, a.ext == SIGN ? N_I2F : N_U2F, a.slot);
    }
    Known k = a;
    switch (to) {
    case T_BOOL:
        if (a.ext == BOTH && a.hi <= 1) return alias(in.dst, a);
        return result(in.dst, bounded(1, to), N_BOOL, a.slot);
    case T_U8: return mask(0xFFu, a.slot, a);
    case T_U16: return mask(0xFFFFu, a.slot, a);
    case T_I32:
        if (k.ext != BOTH) k.ext = SIGN;
        return alias(in.dst, k);
    default:
        if (k.ext != BOTH) {
            k.ext = ZERO;
            k.hi = 0xFFFFFFFFu;
        }
        return alias(in.dst, k);
    }
}

void Translator::one(const xk_vm_ins &in)
{
    const int op = in.op, ty = in.ty;
    if (ty == T_I64 || ty == T_U64 || ty == T_F64) {
        ok = false;
        return;
    }
    switch (op) {
    case 1: {                                              // constant
        const uint64_t v = consts[in.a];
        Known k;
        if (v < (1ull << 31)) k.hi = (uint32_t)v;
        else if (v < (1ull << 32)) k.ext = ZERO, k.hi = 0xFFFFFFFFu;
        else if (v == (uint64_t)(int64_t)(int32_t)(uint32_t)v) k.ext = SIGN, k.hi = 0xFFFFFFFFu;
        else ok = false;
        k.slot = constant((uint32_t)v);
        return alias(in.dst, k);
    }
    case 2: {                                              // parameter
        // its image is checked when it is bound
        params.push_back(XkVmParamUse{in.a, ty == T_I32});
        claim(in.dst);
        emit(N_PARAM, in.dst);
        ops.back().a = in.a;
        reg[in.dst] = bounded(0xFFFFFFFFu, ty);
        reg[in.dst].slot = in.dst;
        return;
    }
    case 3: {                                              // load
        uint64_t hi = g.esz == 1 ? 0xFFull : g.esz == 2 ? 0xFFFFull : 0xFFFFFFFFull;
        if (in.a >= 2 && !g.torus) {
            if (g.border >> 32) ok = false;
            hi = std::max<uint64_t>(hi, g.border & 0xFFFFFFFFull);
        }
        uint32_t imm = 0;
        if (in.a >= 2)
            for (int d = 0; d < g.ndim; ++d) {
                const int delta = g.delta[in.b][d];
                if (delta < -1 || delta > 1) ok = false;
                imm |= (uint32_t)(delta + 1) << (2 * d);
            }
        claim(in.dst);
        emit(N_LOAD, in.dst, -1, -1, -1, imm);
        ops.back().a = in.a >= 2 ? 1 : 0;
        ops.back().b = in.b;
        ops.back().c = in.c;
        reg[in.dst] = bounded(hi, T_U32);
        reg[in.dst].slot = in.dst;
        return;
    }
    case 4: return alias(in.dst, reg[in.a]);
    case 5:
        if (in.b == T_I64 || in.b == T_U64 || in.b == T_F64) ok = false;
        else convert(in);
        return;
    case 30: case 31: case 32: {                           // negation, complement, absolute value
        const Known a = reg[in.a];
        Known f;
        f.ext = ZERO;
        f.hi = 0xFFFFFFFFu;
        if (ty == T_F32) return result(in.dst, f, op == 30 ? N_FNEG : N_FABS, a.slot);
        if (op == 32) {
            if (ty == T_I32 && a.ext == SIGN) return result(in.dst, bounded(0xFFFFFFFFu, ty), N_ABSS, a.slot);
            return alias(in.dst, a);
        }
        if (ty != T_I32 && ty != T_U32) {
            ok = false;
            return;
        }
        return result(in.dst, bounded(0xFFFFFFFFu, ty), op == 30 ? N_NEG : N_NOT, a.slot);
    }
    case 40: {                                             // select
        const Known a = reg[in.a], b = reg[in.b], c = reg[in.c];
        Known k;
        if (b.ext != c.ext && b.ext != BOTH && c.ext != BOTH) ok = false;
        k.ext = b.ext == BOTH ? c.ext : b.ext;
        k.hi = std::max(b.hi, c.hi);
        return result(in.dst, k, N_SEL, a.slot, b.slot, c.slot);
    }
    case 41: {                                             // float bits as int
        Known k = reg[in.a];
        if (k.ext != BOTH) k.ext = SIGN;
        return alias(in.dst, k);
    }
    case 42: {                                             // int bits as float
        Known k = reg[in.a];
        if (k.ext != BOTH) k.ext = ZERO, k.hi = 0xFFFFFFFFu;
        return alias(in.dst, k);
    }
    case 50: return result(in.dst, bounded(32, ty), N_POPC, reg[in.a].slot);
    case 60: return emit(N_STORE, -1, reg[in.a].slot, -1, -1, in.b);
    case 61: return emit(N_COLOR, -1, reg[in.a].slot, reg[in.b].slot, reg[in.c].slot);
    default:
        if (op >= 10 && op <= 25) return binary(in);
        ok = false;
    }
}

// Operations joined with the next one where nothing else reads their result:
// the slot is the next one's result too, or is written before it is read
// again.  Stores of one value one after another become one.
void join(std::vector<XkVnOp> &body)
{
    auto reads = [](const XkVnOp &o, int slot) {
        return ((o.flags & NF_A) && o.a == slot) || ((o.flags & NF_B) && o.b == slot) ||
               ((o.flags & NF_C) && o.c == slot) || ((o.flags & NF_D) && (int)o.imm == slot);
    };
    auto alone = [&](size_t i) {        // only operation i + 1 reads operation i's result
        const int slot = body[i].dst;
        if ((body[i + 1].flags & NF_STORE) && body[i + 1].dst == slot) return true;
        for (size_t k = i + 2; k < body.size(); ++k) {
            if (reads(body[k], slot)) return false;
            if ((body[k].flags & NF_STORE) && body[k].dst == slot) return true;
        }
        return true;
    };
    auto find = [](const int *ops, int n, int op) { return (int)(std::find(ops, ops + n, op) - ops); };
    // the operand of o beside slot (once an operand, first or in an operation
    // that commutes), or -1
    auto other = [](const XkVnOp &o, int slot) {
        if (o.a == slot && o.b != slot) return (int)o.b;
        const bool swaps = o.op == N_ADD || o.op == N_MUL || o.op == N_AND || o.op == N_OR || o.op == N_EQ;
        return o.b == slot && o.a != slot && swaps ? (int)o.a : -1;
    };
    constexpr int FIRSTS = sizeof(VN_FIRST) / sizeof(int);
    std::vector<XkVnOp> out;
    for (size_t i = 0; i < body.size(); ++i) {
        XkVnOp o = body[i];
        const int f = find(VN_FIRST, FIRSTS, o.op);
        if (f < FIRSTS && i + 1 < body.size()) {
            const XkVnOp &p = body[i + 1];
            const int s = find(VN_SECOND, VN_SECONDS, p.op), c = s < VN_SECONDS ? other(p, o.dst) : -1;
            if (c >= 0 && alone(i)) {
                // an addition to the comparison of a masked value
                const int d = o.op == N_AND && p.op == N_EQ && i + 2 < body.size() && body[i + 2].op == N_ADD
                                  ? other(body[i + 2], p.dst) : -1;
                o.c = (uint16_t)c;
                o.flags |= NF_C;
                if (d >= 0 && alone(i + 1)) {
                    o.op = N_COUNT;
                    o.imm = (uint32_t)d;
                    o.flags |= NF_D;
                    o.dst = body[i + 2].dst;
                    i += 2;
                } else {
                    o.op = (uint16_t)(N_PAIR + f * VN_SECONDS + s);
                    o.dst = p.dst;
                    ++i;
                }
            }
        }
        if (o.op == N_STORE && o.imm < 32) {
            uint32_t planes = 1u << o.imm;
            size_t k = i + 1;
            for (; k < body.size() && body[k].op == N_STORE && body[k].a == o.a && body[k].imm < 32; ++k)
                planes |= 1u << body[k].imm;
            if (k > i + 1) {
                o.op = N_STORES;
                o.imm = planes;
                i = k - 1;
            }
        }
        out.push_back(o);
    }
    body.swap(out);
}

}  // namespace

bool xk_vm_translate(const xk_vm_ins *code, int ncode, const uint64_t *consts, int nregs, const VmGeo &g,
                     XkVmNarrow *out)
{
    if (ncode < 1 || g.esz > 4 || g.n > 0x7FFFFFFFll || g.ndim > 8) return false;
    Translator t(consts, nregs, g);
    for (int pc = 0; pc < ncode && t.ok; ++pc) t.one(code[pc]);
    if (!t.ok || t.pool.size() >= XK_VN_CONST) return false;
    std::vector<XkVnOp> &ops = t.ops;
    // Loads before the first store come first, in the program's order, each
    // into a slot of its own; they are numbered after the registers.
    std::vector<XkVnOp> head, body;
    int slots = nregs, colors = 0;
    {
        bool leading = true;
        std::vector<int> now(nregs);
        for (int r = 0; r < nregs; ++r) now[r] = r;
        auto map = [&](uint16_t &s) {
            if (!(s & XK_VN_CONST)) s = (uint16_t)now[s];
        };
        for (XkVnOp o : ops) {
            if (o.flags & NF_A) map(o.a);
            if (o.flags & NF_B) map(o.b);
            if (o.flags & NF_C) map(o.c);
            if (o.op == N_STORE) leading = false;
            if (o.op == N_COLOR) colors = 1;
            if (o.op == N_LOAD && leading) {
                now[o.dst] = slots;
                o.dst = (uint16_t)slots++;
                head.push_back(o);
                continue;
            }
            if (o.flags & NF_STORE) now[o.dst] = o.dst;
            body.push_back(o);
        }
    }
    if (slots >= XK_VN_CONST) return false;
    join(body);
    // slots that are never used drop out
    std::vector<int> used(slots, 0);
    auto mark = [&](const XkVnOp &o) {
        if (o.flags & NF_STORE) used[o.dst] = 1;
        if ((o.flags & NF_A) && !(o.a & XK_VN_CONST)) used[o.a] = 1;
        if ((o.flags & NF_B) && !(o.b & XK_VN_CONST)) used[o.b] = 1;
        if ((o.flags & NF_C) && !(o.c & XK_VN_CONST)) used[o.c] = 1;
        if ((o.flags & NF_D) && !(o.imm & XK_VN_CONST)) used[o.imm] = 1;
    };
    for (const XkVnOp &o : head) mark(o);
    for (const XkVnOp &o : body) mark(o);
    int n = 0;
    for (int &u : used) u = u ? n++ : 0;
    auto renumber = [&](XkVnOp &o) {
        if (o.flags & NF_STORE) o.dst = (uint16_t)used[o.dst];
        if ((o.flags & NF_A) && !(o.a & XK_VN_CONST)) o.a = (uint16_t)used[o.a];
        if ((o.flags & NF_B) && !(o.b & XK_VN_CONST)) o.b = (uint16_t)used[o.b];
        if ((o.flags & NF_C) && !(o.c & XK_VN_CONST)) o.c = (uint16_t)used[o.c];
        if ((o.flags & NF_D) && !(o.imm & XK_VN_CONST)) o.imm = (uint32_t)used[o.imm];
    };
    out->nloads = (int)head.size();
    out->nops = (int)(head.size() + body.size());
    out->nslots = n < 1 ? 1 : n;
    out->colors = colors;
    out->consts = t.pool;
    if (out->consts.empty()) out->consts.push_back(0);
    out->params = t.params;
    // Threads a block: 128, fewer where that leaves SMs without a block or
    // takes more than half an SM's shared memory.
    const int64_t sms = xk_sm_count() > 0 ? xk_sm_count() : 1;
    // the constants' slots follow the registers' and one nothing reads
    const int spare = out->nslots, first = spare + 1;
    out->nslots = first + (int)out->consts.size();
    const int rows = out->nslots + 3 * g.ndim;
    const int64_t threads = (g.n + 3) / 4;
    auto smem = [&](int t) { return (int64_t)rows * t * 16; };
    int T = 128;
    while (T > 32 && (threads / T < 2 * sms || smem(T) > 100 * 1024)) T /= 2;
    if (smem(T) > 200 * 1024) return false;
    out->threads = T;
    out->smem = (int)smem(T);
    out->code.clear();
    auto put = [&](XkVnOp &o) {
        renumber(o);
        XkVnCode c;
        memset(&c, 0, sizeof(c));
        c.op = o.op;
        auto place = [&](int slot) {
            return (uint16_t)(slot & XK_VN_CONST ? first + (slot & (XK_VN_CONST - 1)) : slot);
        };
        // operands an operation does not have read the first constant
        c.dst = (uint16_t)(o.flags & NF_STORE ? o.dst : spare);
        c.a = place(o.flags & NF_A ? o.a : XK_VN_CONST);
        c.b = place(o.flags & NF_B ? o.b : XK_VN_CONST);
        c.c = place(o.flags & NF_C ? o.c : XK_VN_CONST);
        if (o.flags & NF_D) c.plane = place((int)o.imm);
        if (o.op == N_STORE) c.plane = (uint16_t)o.imm;
        if (o.op == N_STORES) c.imm = o.imm;
        if (o.op == N_PARAM) c.c = o.a;
        if (o.op == N_LOAD) {
            c.c = o.a;
            c.plane = o.c;
            c.imm = o.imm;
        }
        out->code.insert(out->code.end(), (const uint32_t *)&c, (const uint32_t *)(&c + 1));
    };
    for (XkVnOp &o : head) put(o);
    for (XkVnOp &o : body) put(o);
    // the two fetched past the end
    XkVnOp none;
    memset(&none, 0, sizeof(none));
    none.op = N_MOV;
    put(none);
    put(none);
    return true;
}

template <int ESZ, class PROG>
static cudaError_t vn_launch(const VnParams &p, const PROG &prog, const XkVmNarrow &v, uint8_t *fld, int32_t *col,
                             cudaStream_t s)
{
    void (*k)(uint8_t *, int32_t *, VnParams, PROG) = xk_k_vm_narrow<ESZ, PROG>;
    if (v.smem > 48 * 1024) {
        const cudaError_t e = xk_smem_attr_at_least((const void *)k, v.smem);
        if (e != cudaSuccess) return e;
    }
    const int64_t cells = 4ll * v.threads;
    return xk_launch_pdl(k, dim3((unsigned)(((int64_t)p.n + cells - 1) / cells)), dim3(v.threads), (size_t)v.smem, s,
                         fld, col, p, prog);
}

// a program that fits an argument of CODE operations and CONSTS constants
template <int ESZ, int CODE, int CONSTS>
static cudaError_t vn_argument(const VnParams &p, const XkVmNarrow &v, uint8_t *fld, int32_t *col, cudaStream_t s)
{
    VnProgram<CODE, CONSTS> prog;
    memcpy(prog.code, v.code.data(), v.code.size() * 4);
    memcpy(prog.consts, v.consts.data(), v.consts.size() * 4);
    return vn_launch<ESZ>(p, prog, v, fld, col, s);
}

template <int ESZ>
static cudaError_t vn_program(const VnParams &p, const XkVmNarrow &v, const uint32_t *code, const uint32_t *consts,
                              uint8_t *fld, int32_t *col, cudaStream_t s)
{
    if (v.nops <= 128 && v.consts.size() <= 64) return vn_argument<ESZ, 128, 64>(p, v, fld, col, s);
    if (xk_vm_narrow_is_argument(v)) return vn_argument<ESZ, 1024, 512>(p, v, fld, col, s);
    const VnProgram<0, 0> prog = {(const XkVnCode *)code, consts};
    return vn_launch<ESZ>(p, prog, v, fld, col, s);
}

cudaError_t xk_vm_run_narrow(const XkVmNarrow &v, const uint32_t *code, const uint32_t *consts,
                             const uint64_t *params, uint8_t *fld, int32_t *col, const VmGeo &g, cudaStream_t s,
                             uint8_t *frame, int frame_smooth)
{
    VnParams p;
    memset(&p, 0, sizeof(p));
    p.params = params;
    p.nloads = v.nloads;
    p.nops = v.nops;
    p.nslots = v.nslots;
    p.nconsts = (int)v.consts.size();
    p.colors = v.colors;
    p.frame = frame;
    p.frame_smooth = frame_smooth;
    p.ndim = g.ndim;
    p.torus = g.torus;
    p.n = (uint32_t)g.n;
    p.border = (uint32_t)g.border;
    for (int d = 0; d < g.ndim; ++d) p.size[d] = (uint32_t)g.size[d];
    p.color_kind = g.color_kind;
    p.fade_in = g.fade_in;
    p.neg_fade_out = (int32_t)(0u - (uint32_t)g.fade_out);
    p.smooth = g.smooth;
    return g.esz == 4 ? vn_program<4>(p, v, code, consts, fld, col, s)
           : g.esz == 2 ? vn_program<2>(p, v, code, consts, fld, col, s)
                        : vn_program<1>(p, v, code, consts, fld, col, s);
}
