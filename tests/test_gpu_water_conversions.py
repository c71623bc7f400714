"""The matrix form of the waters' constraints (configuration preset, mixed
path): its conversions between FP64 and FP32 at the ends of their range."""
import numpy as np
import pytest

from surfactant_enhanced_spreading_gb300 import config_preset as C
from surfactant_enhanced_spreading_gb300 import engine as E

pytestmark = pytest.mark.gpu


def test_a_water_at_rest_stays_at_rest():
    """Rigid waters without velocity or acceleration need no correction: the
    velocities stay exactly zero, the positions where they are."""
    s = C.config_droplet(300, 0, cells=(8, 8, 8), seed=3)
    eng = E.Engine(s, E.MIXED)
    zero = np.zeros_like(s.pos)
    eng.set_state(s.pos, zero, zero, 0.0)
    eng.move_a()
    pos, vel, _ = eng.state()
    assert np.array_equal(pos, s.pos) and np.array_equal(vel, zero)
    eng.force(True, terms=0)
    eng.move_b()
    pos, vel, _ = eng.state()
    assert np.array_equal(pos, s.pos) and np.array_equal(vel, zero)


@pytest.mark.parametrize("speed", [1e40, 1e60, 1e150, np.inf, np.nan])
def test_a_water_beyond_fp32_is_not_finite(speed):
    """One oxygen so fast that its bonds leave FP32's range: no correction
    exists, its water becomes NaN (not some finite place), and the other waters
    keep their bits."""
    s = C.config_droplet(300, 0, cells=(8, 8, 8), seed=4)
    acc = np.zeros_like(s.pos)
    out = []
    for v in (0.0, speed):
        vel = s.vel.copy()
        vel[30, 0] += v
        eng = E.Engine(s, E.MIXED)
        eng.set_state(s.pos, vel, acc, 0.0)
        eng.move_a()
        out.append(eng.state())
    rest = np.ones(s.n_sites, bool)
    rest[30:33] = False
    assert np.isnan(out[1][0][30, 0]) and np.isnan(out[1][1][30, 0])
    for k in (0, 1):
        assert np.array_equal(out[0][k][rest], out[1][k][rest])
