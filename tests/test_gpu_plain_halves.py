"""The plain path's constraint halves: a water over three lanes in small
contexts and on one lane in large ones, surfactants as a wavefront, give the
bits of the sequential sweeps."""
import numpy as np
import pytest

import oracle as O
from surfactant_enhanced_spreading_gb300 import config_preset as C
from surfactant_enhanced_spreading_gb300 import engine as E
from surfactant_enhanced_spreading_gb300 import system as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("preset", [0, 1])
def test_one_and_three_lanes_give_the_same_bits(preset):
    """8,000 waters in the context: a lane each; 301 or 331 alone: three."""
    small = C.config_droplet(331, 5, cells=(8, 8, 8), seed=2) if preset else S.droplet(301, 3, cells=(8, 8, 4), seed=2)
    large = C.config_droplet(7700, 0, cells=(16, 16, 8), seed=3) if preset else S.droplet(7700, 0, cells=(16, 16, 8), seed=3)
    runs = []
    for systems in ([small, large], small):
        eng = E.Engine(systems, E.PLAIN_FP64)
        eng.force(True)
        eng.init_accel()
        eng.run(99101, 3)
        runs.append([a[:small.n_sites] for a in eng.state()] + [eng.etas()[0], eng.failures()[0]])
    for a, b in zip(*runs):
        assert np.array_equal(a, b)


# the last group of 10 waters and the last pair of surfactants part filled;
# maxit small enough that sweeps run out
@pytest.mark.parametrize("water,surf", [(1, 0), (9, 1), (10, 2), (11, 3), (31, 4), (200, 7)])
@pytest.mark.parametrize("maxit", [100, 3, 0])
def test_halves_equal_the_oracle(water, surf, maxit):
    s = S.droplet(water, surf, cells=(8, 8, 4), seed=water + surf)
    rng = np.random.default_rng(7)
    acc = rng.normal(size=s.pos.shape) * (1e-4 / s.masses())[:, None]
    eng = E.Engine(s, E.PLAIN_FP64, shake_maxit=maxit)
    eng.set_state(s.pos, s.vel, acc, 0.0)
    eng.move_a()
    if maxit == 100:
        o = O.Oracle(s)
        o.set(2, acc)
        o.move_a()
        pos, vel, _ = eng.state()
        assert np.array_equal(pos, o.get(0)) and np.array_equal(vel, o.get(1))
    else:   # 1 e-4 is not met in so few sweeps: every molecule but the odd lucky water is counted
        assert water + surf >= eng.failures()[0] >= (surf if maxit else 0) and eng.failures()[0] > 0
