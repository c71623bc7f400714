"""State in and out of the engine on both sides of the size up to which it
goes through mapped host memory (4,096 sites): every value comes back as given."""
import numpy as np
import pytest

from surfactant_enhanced_spreading_gb300 import config_preset as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("water,surf", [(100, 0), (1361, 1), (1365, 0), (1366, 0), (1362, 1)])
def test_state_round_trip(water, surf):
    from surfactant_enhanced_spreading_gb300 import engine as E
    n = C.sheet_cells(water)
    s = C.config_droplet(water, surf, cells=(n, n, C.box_height_cells(water, surf)), seed=5, graphite_layers=2)
    eng = E.Engine(s, E.PLAIN_FP64, device=0)
    rng = np.random.default_rng(water)
    pos = s.pos + rng.normal(scale=1e-3, size=s.pos.shape)
    vel, acc = rng.normal(size=s.pos.shape), rng.normal(size=s.pos.shape)
    eng.set_state(pos, vel, acc, 0.25)
    for got, want in zip(eng.state(), (pos, vel, acc)):
        assert np.array_equal(got, want)
    eng.set_state(vel=acc)                       # one array: the others stay
    for got, want in zip(eng.state(), (pos, acc, acc)):
        assert np.array_equal(got, want)
    f = eng.force(True)
    eng.set_state(acc=vel)
    for got, want in zip(eng.state(), (pos, acc, vel)):
        assert np.array_equal(got, want)
    assert np.isfinite(f).all() and np.array_equal(eng.forces(), f)
