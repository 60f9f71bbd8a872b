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
