"""Cells of up to 64 sites, whose water H targets share the LJ chunk on the FP32
paths: cells around the edges of a pass, and every launch shape alike."""
import numpy as np
import pytest

import oracle as O
from surfactant_enhanced_spreading_gb300 import config_preset as C
from surfactant_enhanced_spreading_gb300 import engine as E
from test_gpu_near_runs import grid_waters, rel

pytestmark = pytest.mark.gpu


# 30, 33, 63 and 66 sites in one cell: one or two targets a lane, whole or parted.  Bar: the mixed paths'
@pytest.mark.parametrize("n", [10, 11, 21, 22])
@pytest.mark.parametrize("precision", [E.MIXED, E.MIXED_COMP])
def test_one_cell(n, precision):
    s = grid_waters(n, 3.1, seed=n)
    assert rel(E.Engine(s, precision).force(True), O.Oracle(s).force(True)) < 1e-5


@pytest.mark.parametrize("precision", [E.MIXED, E.MIXED_COMP])
@pytest.mark.parametrize("water,surf", [(120, 4), (700, 9)])
def test_shapes_give_the_same_bits(precision, water, surf):
    s = C.config_droplet(water, surf, cells=(8, 8, 8), seed=water)
    out = []
    for tile in (32, 64, 128):
        eng = E.Engine(s, precision)
        eng.set_tuning(tile, 2)
        out.append(eng.force(True))
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
