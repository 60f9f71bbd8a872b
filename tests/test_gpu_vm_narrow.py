"""The interpreter's 32-bit form against its general one: random programs of
every operation and 32-bit type, on edge values, run in both forms (one
instruction of a 64-bit type keeps a program on the general form)."""
import ctypes

import numpy as np
import pytest

from xentica_gb300 import _native as nat
from xentica_gb300.core import ir, vm

pytestmark = pytest.mark.gpu

BOOL, U8, U16, I32, U32, I64, F32 = 0, 1, 2, 3, 4, 5, 7
O = vm.OP
EDGE = [0, 1, 2, 3, 7, 31, 32, 33, 127, 255, 256, 65535, 65536, 2 ** 31 - 1, 2 ** 31, 2 ** 31 + 1,
        2 ** 32 - 1, 2 ** 32 - 2]
FLOATS = [0.0, -0.0, 0.5, -0.5, 1.0, -1.0, 255.9, 65536.5, -3.7, 2.5e9, 5e9, -5e9, 1e20, -1e20,
          float("inf"), float("-inf"), float("nan")]


class _Random:
    """A straight-line program whose operands have the types its operations
    name, as the compiler's do, registers reused at random."""

    def __init__(self, seed, nbr, esz, absorb, nregs=24):
        self.r = np.random.RandomState(seed)
        self.nbr, self.esz, self.absorb, self.nregs = nbr, esz, absorb, nregs
        self.code, self.consts, self.types = [], [], {}

    def emit(self, op, ty, a=0, b=0, c=0, result=None):
        dst = int(self.r.randint(self.nregs))
        self.code.append((O[op], ty, dst, a, b, c, 0))
        self.types[dst] = ty if result is None else result

    def pick(self, types):
        regs = [q for q, t in self.types.items() if t in types]
        return int(regs[self.r.randint(len(regs))]) if regs else None

    def load(self):
        kind = int(self.r.randint(4))
        k = int(self.r.randint(self.nbr)) if kind >= 2 else 0
        ty = {1: U8, 2: U16, 4: U32}[self.esz]
        # what the pass does not write in other cells: emit the main plane,
        # absorb the neighbours' buffers and its own planes
        plane = 0 if not self.absorb else int(self.r.randint(1, self.nbr + 1)) if kind >= 2 else \
            int(self.r.randint(self.nbr + 1))
        self.emit("load", ty, kind, k, plane)

    def const(self):
        ty = int(self.r.choice([I32, U32, F32, U8]))
        if ty == F32:
            v = np.float32(FLOATS[self.r.randint(len(FLOATS))])
        elif ty == U8:
            v = int(self.r.randint(256))
        else:
            v = EDGE[self.r.randint(len(EDGE))]
            v = v - 2 ** 32 if ty == I32 and v >= 2 ** 31 else v
        ctype = {I32: ir.I32, U32: ir.U32, F32: ir.F32, U8: ir.U32}[ty]
        self.consts.append(vm.pack_value(v, ctype))
        self.emit("const", ty, len(self.consts) - 1)

    def step(self):
        kind = self.r.randint(12)
        ints = (BOOL, U8, U16, I32, U32)
        if kind == 0:
            return self.const()
        if kind == 1:
            a = self.pick(ints + (F32, ))
            to = int(self.r.choice([BOOL, U8, U16, I32, U32, F32]))
            return self.emit("cvt", to, a, self.types[a])
        if kind == 2:
            a, t = self.pick(ints), int(self.r.choice([I32, U32, F32, U8]))
            b = self.pick((t, ))
            c = self.pick((t, ))
            return self.emit("sel", t, a, b, c) if b is not None else None
        if kind == 3:
            a = self.pick((I32, U32, F32))
            t = self.types[a] if a is not None else None
            op = str(self.r.choice(["neg", "abs"] if t == F32 else ["neg", "~", "abs"]))
            return self.emit(op, t, a) if a is not None else None
        if kind == 4:
            a = self.pick((U32, ))
            return self.emit("popc", I32, a) if a is not None else None
        if kind == 5:
            a = self.pick((I32, U32, F32, U8, U16))
            return self.emit("mov", self.types[a], a)
        t = int(self.r.choice([I32, U32, F32]))
        a, b = self.pick((t, )), self.pick((t, ))
        if a is None:
            return None
        if t == F32:
            op = str(self.r.choice(["+", "-", "*", "/", "<", "<=", ">", ">=", "==", "!="]))
        else:
            op = str(self.r.choice(["+", "-", "*", "/", "%", "&", "|", "^", "<<", ">>", "<", "<=", ">", ">=",
                                    "==", "!="]))
            if op in ("<<", ">>"):
                b = self.pick((I32, ))
                if b is None:
                    return None
        cmp_op = O["<"] <= O[op] <= O["!="]
        return self.emit(op, t, a, b, result=I32 if cmp_op else None)

    def program(self, steps, stores, color):
        for _ in range(3):
            self.load()
            self.const()
        for _ in range(steps):
            self.step()
            if self.r.randint(9) == 0:
                self.load()
        for plane in stores:
            a = self.pick((BOOL, U8, U16, I32, U32, F32))
            self.code.append((O["store"], U32, 0, a, plane, 0, 0))
            self.step()
        if color:
            a, b, c = (self.pick((I32, U32, U8, U16, BOOL)) for _ in range(3))
            self.code.append((O["color"], I32, 0, a, b, c, 0))


def _run(desc, programs, init, col, wide):
    lib = nat.load()
    h = ctypes.c_void_p()
    nat.check(lib.xk_model_create(ctypes.byref(desc), ctypes.byref(h)), "xk_model_create")
    try:
        n = init.size
        for which, p in enumerate(programs):
            code, consts = list(p.code), list(p.consts)
            if wide:
                code.insert(0, (O["const"], I64, p.nregs, 0, 0, 0, 0))
            code = np.array(code, dtype=vm.INS_DTYPE)
            consts = np.array(consts, dtype=np.uint64)
            nat.check(lib.xk_vm_load(h, which, nat.ptr(code), len(code), nat.ptr(consts), len(consts),
                                     p.nregs + 1), "xk_vm_load")
        nat.check(lib.xk_upload(h, nat.ptr(init), n), "xk_upload")
        nat.check(lib.xk_upload_colors(h, nat.ptr(col), n), "xk_upload_colors")
        nat.check(lib.xk_step(h, 3), "xk_step")
        cells, out = np.empty_like(init), np.empty_like(col)
        nat.check(lib.xk_download(h, nat.ptr(cells), n), "xk_download")
        nat.check(lib.xk_download_colors(h, nat.ptr(out), n), "xk_download_colors")
    finally:
        lib.xk_model_destroy(h)
    return cells, out


@pytest.mark.parametrize("seed", range(48))
def test_random_programs(seed):
    r = np.random.RandomState(1000 + seed)
    ndim = int(r.randint(1, 4))
    size = [int(v) for v in r.choice([1, 2, 3, 5, 8, 33, 64], ndim)]
    if seed % 6 == 0:
        size = [257, 41][:ndim] + [2] * (ndim - 2)
    esz = int(r.choice([1, 2, 4]))
    desc = nat.XkDesc()
    desc.abi_version, desc.family, desc.ndim, desc.nbr = nat.XK_ABI_VERSION, nat.XK_FAMILY_VM, ndim, 2 * ndim
    for d, s in enumerate(size):
        desc.size[d] = s
        desc.delta[2 * d][d], desc.delta[2 * d + 1][d] = 1, -1
    desc.torus, desc.state_bytes = int(seed % 2), esz
    desc.border_value = int(r.randint(0, 2 ** min(8 * esz, 31)))
    desc.color_kind = nat.XK_COLOR_MOVING_AVERAGE if seed % 3 else nat.XK_COLOR_PLAIN
    desc.fade_in, desc.fade_out, desc.smooth = 40, 25, 2
    n = int(np.prod(size))
    init = r.choice(np.array(EDGE + [5, 6], dtype=np.uint64), n).astype({1: np.uint8, 2: np.uint16, 4: np.uint32}[esz])
    col = r.randint(-500, 500, 3 * n).astype(np.int32)
    emit = _Random(seed, 2 * ndim, esz, False)
    emit.program(40, range(1, 2 * ndim + 1), False)
    absorb = _Random(7000 + seed, 2 * ndim, esz, True)
    absorb.program(120, [0], True)
    want = _run(desc, (emit, absorb), init, col, True)
    got = _run(desc, (emit, absorb), init, col, False)
    assert np.array_equal(got[0], want[0])
    assert np.array_equal(got[1], want[1])


@pytest.mark.parametrize("ty", [I32, U32])
@pytest.mark.parametrize("swapped", [False, True])
@pytest.mark.parametrize("again", ["never", "after", "overwritten"])
def test_joined_operations(ty, swapped, again):
    """Every pair of operations of which the second reads the first's result,
    on either side, with that result read again, overwritten or dropped; the
    sums of comparisons of masked values; one value stored to several planes."""
    p = type("P", (), {"nregs": 16})()
    p.consts = [vm.pack_value(v, ir.I32 if ty == I32 else ir.U32) for v in (3, 5, 7, 0)]
    code = [(O["load"], U32, 0, 2, 0, 1, 0), (O["load"], U32, 1, 2, 1, 2, 0)]
    code += [(O["const"], ty, 2 + k, k, 0, 0, 0) for k in range(4)]
    code += [(O["cvt"], ty, 0, 0, U32, 0, 0), (O["cvt"], ty, 1, 1, U32, 0, 0), (O["mov"], ty, 6, 5, 0, 0, 0)]
    ops = ["+", "*", "&", "|", "<<", ">>", "==", "<", "<=", "^", "-"]
    for f in ops:
        for s in ops:
            dst = 7 if again == "overwritten" else 8
            code.append((O[f], ty, 7, 0, 2 if f in ("<<", ">>") else 1, 0, 0))
            a, b = (3, 7) if swapped and s not in ("<<", ">>") else (7, 3)
            code.append((O[s], ty, dst, a, b, 0, 0))
            code.append((O["^"], ty, 6, 6, dst, 0, 0))
            if again == "after":
                code.append((O["^"], ty, 6, 6, 7, 0, 0))
            code.append((O["+"], ty, 6, 6, 4, 0, 0))
    for k in range(6):
        code.append((O["&"], ty, 7, k & 1, 2 + k % 3, 0, 0))
        code.append((O["=="], ty, 7 if k & 2 else 8, 7, 2, 0, 0))
        code.append((O["+"], ty, 6, 6, 7 if k & 2 else 8, 0, 0))
    p.code = code + [(O["store"], U32, 0, 6, 0, 0, 0), (O["store"], U32, 0, 6, 0, 0, 0)]
    e = type("P", (), {"nregs": 16, "consts": p.consts})()
    e.code = [(O["load"], U32, 0, 0, 0, 0, 0), (O["const"], U32, 1, 0, 0, 0, 0)]
    e.code += [(O["store"], U32, 0, 0, 1, 0, 0), (O["store"], U32, 0, 0, 3, 0, 0), (O["+"], U32, 2, 0, 1, 0, 0)]
    e.code += [(O["store"], U32, 0, 2, 2, 0, 0), (O["store"], U32, 0, 2, 4, 0, 0)]
    desc = nat.XkDesc()
    desc.abi_version, desc.family, desc.ndim, desc.nbr = nat.XK_ABI_VERSION, nat.XK_FAMILY_VM, 2, 4
    for d, size in enumerate((67, 5)):
        desc.size[d] = size
        desc.delta[2 * d][d], desc.delta[2 * d + 1][d] = 1, -1
    desc.torus, desc.state_bytes, desc.color_kind = 1, 4, nat.XK_COLOR_PLAIN
    r = np.random.RandomState(5)
    init = r.choice(np.array(EDGE, dtype=np.uint64), 67 * 5).astype(np.uint32)
    col = np.zeros(3 * init.size, dtype=np.int32)
    want, got = _run(desc, (e, p), init, col, True), _run(desc, (e, p), init, col, False)
    assert np.array_equal(got[0], want[0])


NONE, WIDE, NARROW, NARROW_LONG = range(4)


class _Model:
    """An interpreted model of two programs, narrow or (wide) held to the
    64-bit form by one instruction of a 64-bit type in each."""

    def __init__(self, desc, programs, init, col, wide=False):
        self.lib, self.n, self.h = nat.load(), init.size, ctypes.c_void_p()
        self.init, self.col = init, col
        nat.check(self.lib.xk_model_create(ctypes.byref(desc), ctypes.byref(self.h)), "xk_model_create")
        assert [self.form(w) for w in (0, 1)] == [NONE, NONE]
        for which, p in enumerate(programs):
            code = ([(O["const"], I64, p.nregs, 0, 0, 0, 0)] if wide else []) + list(p.code)
            code = np.array(code, dtype=vm.INS_DTYPE)
            consts = np.array(p.consts, dtype=np.uint64)
            nat.check(self.lib.xk_vm_load(self.h, which, nat.ptr(code), len(code), nat.ptr(consts), len(consts),
                                          p.nregs + 1), "xk_vm_load")
        nat.check(self.lib.xk_upload(self.h, nat.ptr(init), self.n), "xk_upload")
        nat.check(self.lib.xk_upload_colors(self.h, nat.ptr(col), self.n), "xk_upload_colors")
        if wide:
            assert [self.form(w) for w in (0, 1)] == [WIDE, WIDE]

    def form(self, which):
        return self.lib.xk_vm_form(self.h, which)

    def bind(self, values):
        v = np.array([x % 2 ** 64 for x in values], dtype=np.uint64)
        nat.check(self.lib.xk_vm_set_params(self.h, nat.ptr(v), len(v)), "xk_vm_set_params")

    def step(self, n):
        nat.check(self.lib.xk_step(self.h, n), "xk_step")

    def state(self):
        cells, col = np.empty_like(self.init), np.empty_like(self.col)
        nat.check(self.lib.xk_download(self.h, nat.ptr(cells), self.n), "xk_download")
        nat.check(self.lib.xk_download_colors(self.h, nat.ptr(col), self.n), "xk_download_colors")
        return cells, col

    def frame(self, width, height):
        img = np.empty(3 * width * height, dtype=np.int32)
        nat.check(self.lib.xk_render(self.h, nat.ptr(img), width, height, 1, 0, 0), "xk_render")
        return img.astype(np.uint8)

    def __del__(self):
        self.lib.xk_model_destroy(self.h)


def _same(a, b):
    for x, y in zip(a.state(), b.state()):
        assert np.array_equal(x, y)


def _program(code, consts=(0, ), ty=ir.U32, nregs=16):
    return type("P", (), {"nregs": nregs, "code": code, "consts": [vm.pack_value(v, ty) for v in consts]})()


def _desc(size, esz=4, **fields):
    desc = nat.XkDesc()
    desc.abi_version, desc.family, desc.ndim, desc.nbr = nat.XK_ABI_VERSION, nat.XK_FAMILY_VM, 2, 4
    for d, s in enumerate(size):
        desc.size[d] = s
        desc.delta[2 * d][d], desc.delta[2 * d + 1][d] = 1, -1
    desc.torus, desc.state_bytes, desc.proj_axis1 = 1, esz, 1
    desc.color_kind, desc.fade_in, desc.fade_out, desc.smooth = nat.XK_COLOR_MOVING_AVERAGE, 40, 25, 2
    for k, v in fields.items():
        setattr(desc, k, v)
    return desc


# the main plane into every buffer
COPY = _program([(O["load"], U32, 0, 0, 0, 0, 0)] + [(O["store"], U32, 0, 0, k, 0, 0) for k in range(1, 5)])


# whole blocks of cells and a remainder, rows off 16 bytes, a frame of one row
@pytest.mark.parametrize("size", [(64, 8), (67, 5), (257, 41), (333, 1)])
@pytest.mark.parametrize("kind", [nat.XK_COLOR_MOVING_AVERAGE, nat.XK_COLOR_PLAIN])
@pytest.mark.parametrize("render_smooth", [0, 1, 3])
@pytest.mark.parametrize("scale", [1, 1 << 20])
@pytest.mark.parametrize("where", ["host", "device"])
def test_frames_of_the_absorb_pass(size, kind, render_smooth, scale, where):
    """The zoom-1 frame of the whole lattice, written by the absorb pass:
    colours that are their pixels, and ones beyond 2^24 and below 0, with and
    without a division."""
    desc = _desc(size, color_kind=kind, render_smooth=render_smooth)
    absorb = _program(
        [(O["load"], U32, k, 2, k, k + 1, 0) for k in range(4)] + [(O["load"], U32, 4, 0, 0, 0, 0)] +
        [(O["const"], U32, 5, 0, 0, 0, 0), (O["const"], U32, 6, 1, 0, 0, 0), (O["const"], U32, 12, 2, 0, 0, 0)] +
        [(O["+"], U32, 7, 0, 1, 0, 0), (O["+"], U32, 7, 7, 2, 0, 0), (O["+"], U32, 7, 7, 3, 0, 0)] +
        [(O["^"], U32, 7, 7, 4, 0, 0), (O["&"], U32, 7, 7, 6, 0, 0), (O["store"], U32, 0, 7, 0, 0, 0)] +
        [(O["*"], U32, 8, 7, 5, 0, 0), (O["*"], U32, 9, 4, 5, 0, 0), (O["-"], U32, 10, 12, 8, 0, 0)] +
        [(O["color"], I32, 0, 8, 9, 10, 0)], (scale, 255, 90))
    r = np.random.RandomState(size[0] + scale % 97)
    n = size[0] * size[1]
    init = r.randint(0, 256, n).astype(np.uint32)
    col = r.randint(-100 * scale, 300 * scale, 3 * n).astype(np.int32)
    a, b = _Model(desc, (COPY, absorb), init, col), _Model(desc, (COPY, absorb), init, col, wide=True)
    assert [a.form(w) for w in (0, 1)] == [NARROW, NARROW]
    steps = 6                       # more than the ring of host frames
    want = np.empty((steps, 3 * n), dtype=np.uint8)
    for g in range(steps):
        b.step(1)
        want[g] = b.frame(*size)
    if where == "device":
        torch = pytest.importorskip("torch")
        out = torch.zeros(want.size, dtype=torch.uint8, device="cuda")
        addr = out.data_ptr()
    else:
        out = np.zeros_like(want)
        addr = out.ctypes.data
    nat.check(a.lib.xk_step_frames(a.h, steps, size[0], size[1], 1, 0, 0, ctypes.c_void_p(addr),
                                   int(where == "device")), "xk_step_frames")
    got = out.cpu().numpy().reshape(want.shape) if where == "device" else out
    assert np.array_equal(got, want)
    _same(a, b)


@pytest.mark.parametrize("nops,nconsts", [(128, 64), (129, 30), (100, 65), (1024, 64), (1025, 64), (3000, 300)])
def test_program_lengths(nops, nconsts):
    """Programs at the limits of each kernel argument, and beyond them."""
    consts = [17 * k + 3 for k in range(nconsts - 1)]       # and the 0 of registers nobody wrote
    code = [(O["load"], U32, 1, 0, 0, 0, 0)]
    for k in range(nops - 2):
        code.append((O["const"], U32, 2, k % len(consts), 0, 0, 0))
        code.append((O["-" if k % 2 else "^"], U32, 1, 1, 2, 0, 0))
    absorb = _program(code + [(O["store"], U32, 0, 1, 0, 0, 0)], consts)
    desc = _desc((67, 5), color_kind=nat.XK_COLOR_NONE)
    init = np.random.RandomState(nops).randint(0, 2 ** 32, 67 * 5, dtype=np.uint64).astype(np.uint32)
    col = np.zeros(3 * init.size, dtype=np.int32)
    a, b = _Model(desc, (COPY, absorb), init, col), _Model(desc, (COPY, absorb), init, col, wide=True)
    assert [a.form(w) for w in (0, 1)] == [NARROW, NARROW if nops <= 1024 else NARROW_LONG]
    for m in (a, b):
        m.step(3)
    _same(a, b)


def test_parameters_rebound_in_and_out_of_32_bits():
    """A bound parameter whose image is not the extension of its low half runs
    the 64-bit form until one that is takes its place."""
    absorb = _program(
        [(O["load"], U32, 0, 0, 0, 0, 0), (O["param"], I32, 1, 0, 0, 0, 0), (O["param"], U32, 2, 3, 0, 0, 0)] +
        [(O["const"], I32, 4, 0, 0, 0, 0), (O["<"], I32, 3, 1, 4, 0, 0)] +
        [(O["+"], U32, 5, 0, 2, 0, 0), (O["cvt"], U32, 6, 1, I32, 0, 0)] +
        [(O["/"], U32, 7, 5, 2, 0, 0), (O["^"], U32, 7, 7, 6, 0, 0), (O["+"], U32, 7, 7, 3, 0, 0)] +
        [(O["store"], U32, 0, 7, 0, 0, 0), (O["color"], I32, 0, 3, 7, 1, 0)])
    desc = _desc((33, 9))
    r = np.random.RandomState(2)
    init = r.randint(0, 2 ** 32, 33 * 9, dtype=np.uint64).astype(np.uint32)
    col = r.randint(-500, 500, 3 * init.size).astype(np.int32)
    a, b = _Model(desc, (COPY, absorb), init, col), _Model(desc, (COPY, absorb), init, col, wide=True)
    for first, second, form in [(5, 7, NARROW), (-3, 2 ** 32 - 1, NARROW), (2 ** 40 + 1, 7, WIDE), (5, 7, NARROW),
                                (5, 2 ** 32 + 9, WIDE), (2 ** 31, 1, WIDE), (-2 ** 31, 0, NARROW),
                                (2 ** 31 - 1, 3, NARROW)]:
        for m in (a, b):
            m.bind((first, 0, 2 ** 63, second))
            m.step(2)
        assert [a.form(w) for w in (0, 1)] == [NARROW if form == NARROW else WIDE, form]
        _same(a, b)


@pytest.mark.parametrize("seed", range(24))
def test_random_programs_that_translate(seed):
    """Random programs that the 32-bit form takes (the first of a few draws
    that it does): the form ran, and its cells and colours are the other's."""
    desc = _desc([(64, 33), (5, 7), (1, 130)][seed % 3], [1, 2, 4][seed % 2 + seed % 3 // 2], torus=seed % 2,
                 border_value=77)
    n = desc.size[0] * desc.size[1]
    r = np.random.RandomState(300 + seed)
    init = r.randint(0, 200, n).astype({1: np.uint8, 2: np.uint16, 4: np.uint32}[desc.state_bytes])
    col = r.randint(-500, 500, 3 * n).astype(np.int32)
    for draw in range(30):
        emit = _Random(100 * seed + draw, 4, desc.state_bytes, False)
        emit.program(12, range(1, 5), False)
        absorb = _Random(70000 + 100 * seed + draw, 4, desc.state_bytes, True)
        absorb.program(50, [0], True)
        a = _Model(desc, (emit, absorb), init, col)
        if [a.form(w) for w in (0, 1)] == [NARROW, NARROW]:
            break
    else:
        pytest.fail("no draw translated")
    b = _Model(desc, (emit, absorb), init, col, wide=True)
    for m in (a, b):
        m.step(3)
    _same(a, b)
