"""A negative sweep limit: the constraint halves of every precision make no sweep,
count every molecule as failed and return."""
import numpy as np
import pytest

from surfactant_enhanced_spreading_gb300 import config_preset as C
from surfactant_enhanced_spreading_gb300 import engine as E
from surfactant_enhanced_spreading_gb300 import system as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("preset", [0, 1])
@pytest.mark.parametrize("precision", [E.PLAIN_FP64, E.MIXED, E.MIXED_FP32C, E.MIXED_COMP])
def test_no_sweep_is_a_failure(precision, preset):
    s = C.config_droplet(40, 3, cells=(8, 8, 8), seed=2) if preset else S.droplet(40, 3, cells=(8, 8, 4), seed=2)
    constrained = 40 if preset else 43          # the configuration preset's chains have no constraints
    eng = E.Engine(s, precision, shake_maxit=-1)
    eng.set_state(s.pos, s.vel, np.zeros_like(s.pos), 0.0)
    eng.move_a()
    assert eng.failures()[0] == constrained
    eng.force(True, terms=0)
    eng.move_b()
    assert eng.failures()[0] == 2 * constrained
