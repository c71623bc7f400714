"""Far field of the plain path with classes of 256 occupied cells and more,
whose tiles take a target per lane: classes below, at and above that, and last
tiles of a part."""
import numpy as np
import pytest

import oracle as O
from surfactant_enhanced_spreading_gb300 import engine as E
from test_gpu_far_lists import scattered

pytestmark = pytest.mark.gpu


# 2,048 cells are 256 a class; bar: FP64 rounding
@pytest.mark.parametrize("used,cells", [(2030, (16, 16, 8)), (2048, (16, 16, 8)), (2100, (16, 16, 12)), (3072, (16, 16, 12)),
                                        (9216, (24, 24, 16))])
def test_many_targets(used, cells):
    s = scattered(used, cells, used)
    fo = O.Oracle(s).force(True, terms=E.T_FAR)
    assert np.linalg.norm(E.Engine(s, E.PLAIN_FP64).force(True, terms=E.T_FAR) - fo) < 1e-10 * np.linalg.norm(fo)
