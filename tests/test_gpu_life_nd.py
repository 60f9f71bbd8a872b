"""Bit-packed N-D Life-like lattices against the oracle, cell by cell: widths
around a word's edges, axes of one and two cells (a neighbour met twice), both
borders, every count width (3, 4 and 5 planes)."""
import numpy as np
import pytest

import oracle as O
from tests.models import GOLExperiment2, LifelikeFixed
from xentica_gb300 import core

pytestmark = pytest.mark.gpu


def _model(kind, ndim, border):
    topo = type("Topology", (), {
        "dimensions": ndim, "lattice": core.OrthogonalLattice(),
        "neighborhood": core.MooreNeighborhood() if kind == "moore" else core.VonNeumannNeighborhood(),
        "border": core.TorusBorder() if border is None else core.StaticBorder(border)})
    return type(core.CellularAutomaton)("NdLife", (LifelikeFixed, ), {"Topology": topo, "state": core.IntegerProperty(max_val=1)})


CASES = [("moore", size, border)
         for size in ((1, 1, 1), (2, 2, 3), (31, 3, 2), (32, 5, 1), (33, 4, 6), (64, 7, 5), (65, 33, 3), (96, 2, 17))
         for border in (None, 0, 1)]
CASES += [("von_neumann", size, border)
          for size in ((1, ), (77, ), (33, 10), (64, 3), (32, 5, 4), (70, 9, 1), (5, 3, 4, 6), (34, 3, 2, 2),
                       (3, 3, 4, 3, 3, 4), (33, 2, 1, 2, 3, 1, 2))
          for border in (None, 1)]
CASES += [("moore", (40, ), None), ("moore", (40, ), 1)]


@pytest.mark.parametrize("kind,size,border", CASES)
def test_against_oracle(kind, size, border):
    rng = np.random.RandomState(sum(size) + len(size))
    rule = int(rng.randint(0, 2 ** 31 - 1))
    exp = type("E", (GOLExperiment2, ), {"size": size, "rule": rule})
    model = _model(kind, len(size), border)(exp)
    topo = O.Topology(size, kind, border)
    fld = topo.field(model.gpu.arrays.cells.get()[:model.cells_num], np.uint8)
    col = np.zeros(topo.cells * 3, dtype=np.int32)
    # the rule as the model's absorb reads it: counts above 8 see the survival bits
    for _ in range(5):
        model.step()
        O.life_run(topo, fld, col, 1, born=rule, sustain=rule >> 9)
        assert np.array_equal(model.gpu.arrays.cells.get()[:model.cells_num], fld[:topo.cells])
    model.gpu.step(4)
    O.life_run(topo, fld, col, 4, born=rule, sustain=rule >> 9)
    assert np.array_equal(model.gpu.arrays.cells.get()[:model.cells_num], fld[:topo.cells])
    assert np.array_equal(model.gpu.arrays.colors.get(), col)


# 3-D von Neumann lattices on clusters of 1 to 16 CTAs (fewer planes than
# CTAs, slabs of unequal planes, planes of more words than threads), and one
# that no cluster holds
@pytest.mark.parametrize("size", [(1, 1, 1), (33, 9, 1), (64, 40, 2), (256, 130, 3), (64, 64, 13), (67, 66, 65),
                                  (256, 256, 20), (155, 141, 55), (192, 180, 190), (256, 200, 256)])
@pytest.mark.parametrize("border", [None, 0, 1])
def test_faces_against_oracle(size, border):
    rng = np.random.RandomState(sum(size))
    rule = 4 | 12 << 9 if border == 0 else int(rng.randint(0, 2 ** 31 - 1))
    exp = type("E", (GOLExperiment2, ), {"size": size, "rule": rule})
    model = _model("von_neumann", 3, border)(exp)
    n = model.cells_num
    cells = (rng.random_sample(n) < 0.3).astype(np.uint8)
    model.gpu.load(cells, np.zeros(3 * n, dtype=np.int32))
    topo = O.Topology(size, "von_neumann", border)
    fld = topo.field(cells, np.uint8)
    col = np.zeros(topo.cells * 3, dtype=np.int32)
    for k in (1, 11, 2):
        model.gpu.step(k)
        O.life_run(topo, fld, col, k, born=rule, sustain=rule >> 9)
        assert np.array_equal(model.gpu.arrays.cells.get()[:n], fld[:n]), k
