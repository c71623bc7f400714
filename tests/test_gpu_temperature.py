"""The temperature of one, of as many replicas as fit the mapped result
buffer (256), and of one more, whose sums are copied back."""
import pytest

from surfactant_enhanced_spreading_gb300 import engine as E
from surfactant_enhanced_spreading_gb300 import initial as I
from surfactant_enhanced_spreading_gb300 import system as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("replicas", [1, 256, 257])
def test_temperature_of_many_replicas(replicas):
    s = S.droplet(60, 1, cells=(4, 4, 4), seed=9)
    eng = E.Engine([s] * replicas, E.MIXED)
    want = I.temperature(s.vel, s.n_water, s.n_surf)
    got = [eng.temperature(), eng.temperature()]   # the second: the slice counters are back at 0
    eng.set_state(None, 2.0 * eng.state()[1], None, 0.0)
    got.append(eng.temperature() / 4.0)
    # both sums have fewer than 1e5 positive terms in FP64
    assert all(abs(t - want) < 1e-11 * want for t in got)
