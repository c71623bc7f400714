"""The scan over cells on both sides of 65,536 of them, from where it goes in two
launches: a replica's forces do not depend on the context's size."""
import dataclasses

import numpy as np
import pytest

from surfactant_enhanced_spreading_gb300 import config_preset as C
from surfactant_enhanced_spreading_gb300 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("replicas", [127, 128, 129, 260])
def test_many_cells(replicas):
    """Replicas of 512 cells: 65,024, 65,536, 66,048 and 133,120 cells."""
    kinds = [C.config_droplet(n, n // 40, cells=(8, 8, 8), seed=n, graphite_layers=0) for n in (40, 61, 90)]
    alone = [E.Engine(s, E.MIXED).force(True) for s in kinds]
    eng = E.Engine([dataclasses.replace(kinds[k % 3]) for k in range(replicas)], E.MIXED)
    f = eng.force(True)
    for k in range(replicas):
        assert np.array_equal(f[eng.offsets[k]:eng.offsets[k + 1]], alone[k % 3])
    checks = eng.checks()
    assert (checks[:, 6] == 0).all() and (checks[:, 7] == 0).all()
