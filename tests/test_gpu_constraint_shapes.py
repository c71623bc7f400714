"""Mixed path: a surfactant's sweeps run 4 steps apart alone in a warp and 6
steps apart two to a warp, and stop after maxit + 1; the state has the same
bits."""
import numpy as np
import pytest

from surfactant_enhanced_spreading_gb300 import engine as E
from surfactant_enhanced_spreading_gb300 import system as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("surf", [1, 2, 3, 7])
@pytest.mark.parametrize("maxit", [100, 5, 3, 1, 0, -1])
def test_one_and_two_a_warp(surf, maxit):
    s = S.droplet(20, surf, cells=(8, 8, 4), seed=surf)
    acc = np.random.default_rng(7).normal(size=s.pos.shape) * (1e-4 / s.masses())[:, None]
    out = []
    for mols in (1, 2):
        eng = E.Engine(s, E.MIXED, shake_maxit=maxit)
        eng.set_constraint_tuning(2, mols)
        eng.set_state(s.pos, s.vel, acc, 0.0)
        eng.move_a()
        after = list(eng.state()) + [eng.failures()]
        eng.set_state(s.pos, s.vel, acc, 0.0)      # RATTLE from the same state, with no force
        eng.force(True, terms=0)
        eng.move_b()
        out.append(after + [eng.state()[1], eng.failures() - after[3]])
    one, two = out
    for a, b in zip(one, two):
        assert np.array_equal(a, b)
    if maxit < 0:
        assert one[3][0] == one[5][0] == 20 + surf
