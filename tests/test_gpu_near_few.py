"""FP32 pair fields of cells with few sites and partners, which are one item per
plane of their shell: thin gases of waters and of chains or surfactants, on both
sides of the rule's limits, against the oracle and in every context and launch
shape alike."""
import dataclasses

import numpy as np
import pytest
from scipy.spatial import cKDTree

import oracle as O
from surfactant_enhanced_spreading_gb300 import config_preset as C
from surfactant_enhanced_spreading_gb300 import engine as E
from surfactant_enhanced_spreading_gb300 import system as S
from test_gpu_near_runs import rel

pytestmark = pytest.mark.gpu


def lattice(n, low, high, rng):
    k = np.ceil((high - low) * (n / np.prod(high - low)) ** (1 / 3)).astype(int)
    g = np.stack(np.meshgrid(*[np.linspace(low[a], high[a], max(k[a], 2)) for a in range(3)], indexing="ij"), -1).reshape(-1, 3)
    return g[np.sort(rng.permutation(len(g))[:n])] + rng.uniform(-0.1, 0.1, (n, 3))


def gas(preset, water, surf, cells, seed, kept=1.0):
    """A droplet's molecules on jittered lattices over the lower part `kept` of
    the box, without the waters closer than 3 A to a surfactant."""
    s = (C.config_droplet(water, surf, cells=(8, 8, 8), seed=seed, graphite_layers=0) if preset
         else S.droplet(water, surf, cells=(8, 8, 8), seed=seed, graphite_layers=0))
    rng = np.random.default_rng(seed)
    half = np.array(cells) * S.RS / 2
    wat, sur = s.pos[:3 * water].reshape(water, 3, 3), s.pos[3 * water:].reshape(surf, s.sites_per_surf, 3)
    wat = wat - wat.mean(1, keepdims=True) + lattice(water, 2.5 - half, (half - 2.5) * [1, 1, 2 * kept - 1], rng)[:, None]
    if surf:
        sur = sur - sur.mean(1, keepdims=True) + lattice(surf, 6.5 - half, half - 6.5, rng)[:, None]
        wat = wat[cKDTree(sur.reshape(-1, 3)).query(wat.reshape(-1, 3))[0].reshape(-1, 3).min(1) > 3.0 / S.SIGMA]
    pos = np.concatenate([wat.reshape(-1, 3), sur.reshape(-1, 3)])
    return dataclasses.replace(s, n_water=len(wat), cells=tuple(cells), pos=pos, vel=np.zeros_like(pos))


# about 1/3, 1, 2, 3, 4 and 6 waters a cell (6 turns a plane and 24 sites a cell
# are the limits); surfactants of 12 or 29 sites in
# place of some.  Bar: the mixed paths'
@pytest.mark.parametrize("preset", [0, 1])
@pytest.mark.parametrize("water,surf", [(170, 0), (512, 0), (1024, 0), (1500, 0), (2048, 0), (3000, 0), (150, 12), (600, 20)])
def test_gas(preset, water, surf):
    s = gas(preset, water, surf, (8, 8, 8), seed=water)
    fo = O.Oracle(s).force(True, terms=O.TERM_NEAR)
    assert rel(E.Engine(s, E.MIXED).force(True, terms=E.T_NEAR), fo) < 1e-5
    assert rel(E.Engine(s, E.MIXED_COMP).force(True, terms=E.T_NEAR), fo) < 1e-5


@pytest.mark.parametrize("precision", [E.MIXED, E.MIXED_COMP])
@pytest.mark.parametrize("preset", [0, 1])
def test_any_context_and_shape(precision, preset):
    """Alone the gas runs by single cells, in a batch of 16,000 sites by rows; the bits are the same."""
    s = gas(preset, 700, 20, (8, 8, 8), seed=3, kept=0.6)
    other = gas(preset, 5000, 0, (12, 12, 8), seed=4)
    alone = E.Engine(s, precision)
    f = alone.force(True)
    assert np.array_equal(E.Engine([s, other], precision).force(True)[:s.n_sites], f)
    for tile in (32, 128):
        alone.set_tuning(tile, 2)
        assert np.array_equal(alone.force(True), f)
        assert np.array_equal(alone.force(False), f)
