"""Plain path: a site far from its frozen cell takes only its own neighbours'
blocks of pairs off the fixed-point arithmetic."""
import numpy as np
import pytest

from surfactant_enhanced_spreading_gb300 import config_preset as C
from surfactant_enhanced_spreading_gb300 import engine as E
from surfactant_enhanced_spreading_gb300 import system as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("drift", [2.8, 1e3, np.inf, np.nan])
@pytest.mark.parametrize("preset", [0, 1])
def test_other_sites_keep_their_bits(preset, drift):
    """One hydrogen moved off along frozen lists: sites whose cells are not
    next to its own have the same force to the last bit."""
    s = (C.config_droplet(900, 9, cells=(8, 8, 8), seed=4) if preset else S.droplet(900, 6, cells=(8, 8, 8), seed=4))
    eng = E.Engine(s, E.PLAIN_FP64)
    f0 = eng.force(True, terms=E.T_NEAR)
    half = 4 * S.RS
    cell = np.floor((s.pos + half) / S.RS).astype(int)
    gap = np.abs(cell - cell[1])
    if preset:
        gap[:, :2] = np.minimum(gap[:, :2], 8 - gap[:, :2])
    apart = gap.max(axis=1) > 1
    assert 100 < apart.sum() < s.n_sites
    pos = s.pos.copy()
    # away from its cell's centre: beyond the reach of 2.7 sigma
    pos[1, 0] += drift * (1.0 if s.pos[1, 0] + half - (cell[1, 0] + 0.5) * S.RS > 0 else -1.0)
    eng.set_state(pos)
    f1 = eng.force(False, terms=E.T_NEAR)
    assert np.array_equal(f1[apart], f0[apart])
    eng.set_state(s.pos)
    assert np.array_equal(eng.force(False, terms=E.T_NEAR), f0)
