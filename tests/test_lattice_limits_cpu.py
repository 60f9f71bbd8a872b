"""Index arithmetic of the kernels at the widest lattices a model accepts
(sides up to 2^31 - 1 cells).

The functions that the kernels and their launchers share are compiled as host
code with nvcc (no GPU needed) and checked against 64-bit arithmetic.
"""
import os
import subprocess

import pytest

from tests.test_div_magic_cpu import CSRC, INCLUDE, _nvcc


def _run(tmp_path, program):
    nvcc = _nvcc()
    if not nvcc:
        pytest.skip("nvcc not found")
    src, exe = str(tmp_path / "limits.cu"), str(tmp_path / "limits")
    with open(src, "w") as fh:
        fh.write(program)
    subprocess.run([nvcc, "-std=c++17", "-O2", "-I", CSRC, "-I", INCLUDE, src, "-o", exe],
                   check=True, capture_output=True, text=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()


def test_halves_of_a_rows_last_word(tmp_path):
    """Rows of a multiple of 16 cells, up to 2^31 - 16: every word but an odd
    row's last one has two halves."""
    out = _run(tmp_path, r"""
#include "xk_internal.cuh"
#include <cstdio>

int main()
{
    long long checked = 0, bad = 0;
    for (int64_t W : {16ll, 32ll, 48ll, 1024ll, 1040ll, (1ll << 30) + 16, (1ll << 31) - 48, (1ll << 31) - 32,
                      (1ll << 31) - 16}) {
        const int64_t words = (W + 31) / 32;
        for (int64_t j : {(int64_t)0, words / 2, words - 2, words - 1}) {
            if (j < 0) continue;
            ++checked;
            bad += xk_word_halves((uint32_t)j, (int32_t)W) != (32 * j + 32 <= W ? 2 : 1);
        }
    }
    std::printf("%lld %lld\n", checked, bad);
}
""")
    assert int(out[0]) > 30 and int(out[1]) == 0


@pytest.mark.parametrize("tile,halo", [(120, 4)])
def test_columns_of_a_tile(tmp_path, tile, halo):
    """Every column of the first and the last two tiles of a row, rows of one
    cell to 2^31 - 1, as a kernel forms it modulo 2^32: inside the row or not,
    and the wrapped one."""
    out = _run(tmp_path, r"""
#include "xk_internal.cuh"
#include <cstdio>

int main()
{
    const int64_t tile = %d, halo = %d;
    long long checked = 0, bad = 0;
    for (int64_t W : {1ll, 2ll, 3ll, 5ll, 119ll, 120ll, 121ll, 123ll, 240ll, 1000ll, (1ll << 31) - 250,
                      (1ll << 31) - 129, (1ll << 31) - 128, (1ll << 31) - 64, (1ll << 31) - 9, (1ll << 31) - 1}) {
        const int64_t tiles = (W + tile - 1) / tile;
        for (int64_t t : {(int64_t)0, tiles - 2, tiles - 1})
            for (int64_t off = -halo; off < tile + halo; ++off) {
                if (t < 0) continue;
                const int64_t x = t * tile + off, wrapped = ((x %% W) + W) %% W;
                const uint32_t xu = (uint32_t)(t * tile) + (uint32_t)off;
                const bool in = xu < (uint32_t)W;
                ++checked;
                bad += in != (x >= 0 && x < W) || (in ? (int)xu : xk_wrap_column(xu, (int)W)) != wrapped;
            }
    }
    std::printf("%%lld %%lld\n", checked, bad);
}
""" % (tile, halo))
    assert int(out[0]) > 4000 and int(out[1]) == 0


@pytest.mark.parametrize("side", [60, 64, 30, 16])
def test_tiles_in_range(tmp_path, side):
    """Where the rule for tiles holds, the farthest cell that the last tile
    looks at (its start, its side, its halo, the cells loaded beside it: up to
    64 on from its start, or 40 beyond it in rows) is an int; ordinary sides
    are in range."""
    out = _run(tmp_path, r"""
#include "xk_internal.cuh"
#include <cstdio>

int main()
{
    const int64_t side = %d;
    long long in = 0, bad = 0;
    for (int64_t n = (1ll << 31) - 200; n < 1ll << 31; ++n) {
        const int64_t start = (n - 1) / side * side;
        if (!xk_tiles_in_range(n, 1) || !xk_tiles_in_range(1, n)) continue;
        ++in;
        bad += start + 64 > 0x7FFFFFFFll || n + side - 1 > 0x7FFFFFFFll;
    }
    std::printf("%%lld %%lld %%d\n", in, bad, (int)xk_tiles_in_range((1ll << 31) - 200, 1 << 30));
}
""" % side)
    assert int(out[0]) > 100 and int(out[1]) == 0 and out[2] == "1"
