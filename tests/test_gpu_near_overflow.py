"""The FP32 pair fields with a site so far off on frozen lists that its squared
distances overflow FP32: it exerts no force, and the others keep theirs."""
import numpy as np
import pytest

from surfactant_enhanced_spreading_gb300 import config_preset as C
from surfactant_enhanced_spreading_gb300 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,bar", [(E.MIXED, 1e-5), (E.MIXED_COMP, 1e-5)])
@pytest.mark.parametrize("drift", [1e6, 1.3e19, 1e20, 1e25])
def test_a_site_out_of_range_spoils_no_other(precision, bar, drift):
    """Against the same site 1e6 sigma away, whose Coulomb force (1e-12 of a
    neighbour's) is far below the mixed paths' bar."""
    s = C.config_droplet(600, 8, cells=(8, 8, 8), seed=9)
    for moved in (30, 31, 3 * s.n_water + 2):      # a water O, a water H, a bead
        eng = E.Engine(s, precision)
        eng.force(True, terms=E.T_NEAR)
        f = []
        for d in (1e6, drift):
            pos = s.pos.copy()
            pos[moved, 0] += d
            eng.set_state(pos)
            f.append(eng.force(False, terms=E.T_NEAR))
        rest = np.arange(s.n_sites) != moved
        assert np.isfinite(f[1]).all()
        assert np.linalg.norm((f[1] - f[0])[rest]) < bar * np.linalg.norm(f[0][rest])
