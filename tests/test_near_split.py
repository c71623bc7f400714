"""Up to which size the pair field's items are single cells: the server's memory
estimate follows the library's constants and stays an upper one."""
import os
import re

import pytest

from surfactant_enhanced_spreading_gb300 import config_preset as C
from surfactant_enhanced_spreading_gb300 import engine as E
from surfactant_enhanced_spreading_gb300 import serve

CSRC = os.path.join(os.path.dirname(E.__file__), "csrc", "sesp_api.cu")


def test_constants_are_the_librarys():
    with open(CSRC) as f:
        m = re.search(r"constexpr int NEAR_SPLIT_MAX = (\d+), NEAR_SPLIT_MAX64 = (\d+);", f.read())
    assert (serve.NEAR_SPLIT_MAX, serve.NEAR_SPLIT_MAX64) == (int(m[1]), int(m[2]))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [E.PLAIN_FP64, E.MIXED, E.MIXED_FP32C, E.MIXED_COMP])
@pytest.mark.parametrize("side", [0, 1])
def test_estimate_is_an_upper_one(precision, side):
    limit = serve.NEAR_SPLIT_MAX64 if precision == E.PLAIN_FP64 else serve.NEAR_SPLIT_MAX
    water = limit // 3 + side
    n = C.sheet_cells(water)
    s = C.config_droplet(water, 0, cells=(n, n, C.box_height_cells(water, 0)), seed=1, graphite_layers=2)
    assert (s.n_sites <= limit) == (side == 0)
    eng = E.Engine(s, precision)
    assert eng.device_bytes() <= serve.estimate_bytes(s, precision) <= serve.estimate_bytes(s)
