"""The far field runs over lists of the occupied boxes: tiles of a class's
targets around their sizes, and boxes that fill and empty between rebuilds."""
import numpy as np
import pytest

import oracle as O
from surfactant_enhanced_spreading_gb300 import config_preset as C
from surfactant_enhanced_spreading_gb300 import engine as E
from surfactant_enhanced_spreading_gb300 import system as S

pytestmark = pytest.mark.gpu


def scattered(n_cells_used, cells, seed):
    """One water in each of `n_cells_used` cells drawn without replacement."""
    rng = np.random.default_rng(seed)
    c = rng.choice(int(np.prod(cells)), n_cells_used, replace=False)
    idx = np.stack([c % cells[0], c // cells[0] % cells[1], c // (cells[0] * cells[1])], 1)
    s = C.config_droplet(max(n_cells_used, 200), 0, cells=cells, seed=0, graphite_layers=0)
    o = (idx + 0.5) * S.RS - s.half_box + rng.uniform(-1, 1, (n_cells_used, 3))
    wat = np.einsum("ij,mkj->mik", S.water_template() / S.SIGMA, S._rand_rots(rng, n_cells_used)) + o[:, None, :]
    return S.System(n_water=n_cells_used, n_surf=0, cells=cells, pos=wat.reshape(-1, 3),
                    vel=np.zeros((3 * n_cells_used, 3)), carbons=np.zeros((0, 3)), graphite_on=False, preset=1)


# occupied cells per parity class: 1 or none, around 16 (128 cells), several
# tiles, all 64 of a class in 8 x 8 x 8 cells.  Bars: the far field alone to
# FP64 rounding, and FP32's 1e-5 of the mixed path.
@pytest.mark.parametrize("used,cells", [(3, (8, 8, 8)), (100, (8, 8, 8)), (128, (8, 8, 8)), (150, (8, 8, 8)),
                                        (512, (8, 8, 8)), (700, (12, 8, 12)), (1500, (16, 16, 8))])
def test_occupied_targets(used, cells):
    s = scattered(used, cells, used)
    o = O.Oracle(s)
    fo = o.force(True, terms=E.T_FAR)
    assert np.linalg.norm(E.Engine(s, E.PLAIN_FP64).force(True, terms=E.T_FAR) - fo) < 1e-10 * np.linalg.norm(fo)
    assert np.linalg.norm(E.Engine(s, E.MIXED).force(True, terms=E.T_FAR) - fo) < 1e-5 * np.linalg.norm(fo)


@pytest.mark.parametrize("precision", [E.PLAIN_FP64, E.MIXED])
@pytest.mark.parametrize("preset", [0, 1])
def test_boxes_fill_and_empty(preset, precision):
    """A rebuild after the droplet has moved three cells along gives the bits
    of an engine that never saw it elsewhere."""
    s = C.config_droplet(300, 3, cells=(12, 8, 8), seed=4) if preset else S.droplet(300, 3, cells=(12, 8, 8), seed=4)
    shift = np.array([3 * S.RS if preset else 1.5 * S.RS, 0.0, 0.0])
    start, moved = s.pos - shift, s.pos + shift
    eng = E.Engine(S.dataclasses.replace(s, pos=start), precision)
    f0 = eng.force(True)
    eng.set_state(moved)
    f1 = eng.force(True)
    assert np.array_equal(f1, E.Engine(S.dataclasses.replace(s, pos=moved), precision).force(True))
    eng.set_state(start)
    assert np.array_equal(eng.force(True), f0)
