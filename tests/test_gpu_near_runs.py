"""The pair field over a partner cell's runs (water O, other LJ sites, water
H, each in groups of four): chunk and run edges, cells of several staged
blocks, an overflowing cell, and items of single cells against rows of
three."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from surfactant_enhanced_spreading_gb300 import config_preset as C
from surfactant_enhanced_spreading_gb300 import engine as E
from surfactant_enhanced_spreading_gb300 import system as S

pytestmark = pytest.mark.gpu


def grid_waters(n, spacing, seed=0):
    """n waters on a cubic grid from the corner of one cell, in Angstrom spacing."""
    s = C.config_droplet(max(n, 200), 0, cells=(8, 8, 8), seed=seed, graphite_layers=0)
    rng = np.random.default_rng(seed)
    k = int(np.ceil(n ** (1.0 / 3.0)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * spacing + 1.1
    wat = np.einsum("ij,mkj->mik", S.water_template(), S._rand_rots(rng, n)) + g[:, None, :]
    return dataclasses.replace(s, n_water=n, pos=wat.reshape(-1, 3) / S.SIGMA, vel=np.zeros((3 * n, 3)))


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# targets and partners of one cell around the 4, 32 and 64 edges of runs and
# chunks; 100 waters in one cell are 75 groups: two staged blocks.  Bars: the
# parity bars of the plain and the mixed paths.
@pytest.mark.parametrize("n,spacing", [(1, 3.0), (2, 3.0), (3, 3.0), (8, 3.1), (15, 3.1), (16, 3.1), (17, 3.1), (31, 3.1),
                                       (32, 3.1), (33, 2.7), (64, 2.7), (65, 2.3), (100, 2.3)])
def test_one_cell_of_waters(n, spacing):
    s = grid_waters(n, spacing, seed=n)
    fo = O.Oracle(s).force(True)
    for mode, bar in ((E.PLAIN_FP64, 1e-10), (E.MIXED, 1e-5), (E.MIXED_COMP, 1e-5)):
        f = E.Engine(s, mode).force(True)
        if n == 1:
            assert np.abs(f - fo).max() <= bar * 1e3   # no partner: only the walls' ~0 force
        else:
            assert rel(f, fo) < bar, mode


# chains and surfactants: the runs with a charge per partner
@pytest.mark.parametrize("preset,water,surf", [(1, 40, 1), (1, 129, 7), (1, 700, 14), (0, 50, 1), (0, 333, 5)])
def test_runs_with_surfactants(preset, water, surf):
    s = (C.config_droplet(water, surf, cells=(8, 8, 8), seed=water) if preset
         else S.droplet(water, surf, cells=(8, 8, 8), seed=water))
    fo = O.Oracle(s).force(True)
    assert rel(E.Engine(s, E.PLAIN_FP64).force(True), fo) < 1e-10
    assert rel(E.Engine(s, E.MIXED).force(True), fo) < 1e-5
    assert rel(E.Engine(s, E.MIXED_COMP).force(True), fo) < 1e-5


def test_overflowing_cell():
    """More sites in a cell than the sort holds (2,048): every slot takes its
    own charge and kind.  Sites of different molecules nearly touch there, so
    the mixed bar is FP32's rounding of the coordinates (2e-7 sigma) against
    the nearest distances (some 0.02 sigma), times LJ's 13th power."""
    s = grid_waters(700, 1.2, seed=3)
    fo = O.Oracle(s).force(True)
    assert rel(E.Engine(s, E.PLAIN_FP64).force(True), fo) < 1e-10
    assert rel(E.Engine(s, E.MIXED).force(True), fo) < 2e-4


@pytest.mark.parametrize("precision", [E.PLAIN_FP64, E.MIXED, E.MIXED_COMP])
def test_cells_and_rows_give_the_same_bits(precision):
    """A small system alone runs single cells as items, in a large batch rows
    of three: its forces are the same."""
    small = C.config_droplet(600, 9, cells=(8, 8, 8), seed=5)
    large = C.config_droplet(13600, 0, cells=(16, 16, 8), seed=6)
    batch = E.Engine([small, large], precision)
    assert batch.n > 40000 > small.n_sites
    fb = batch.force(True)
    assert np.array_equal(fb[:small.n_sites], E.Engine(small, precision).force(True))


@pytest.mark.parametrize("precision,bar", [(E.PLAIN_FP64, 1e-10), (E.MIXED, 1e-5)])
@pytest.mark.parametrize("drift", [0.5, 0.79, 0.81, 1.7, 40.0])
def test_sites_that_leave_their_cells(drift, precision, bar):
    """Frozen lists with every third molecule moved `drift` sigma along x: the
    FP64 path's fixed-point coordinates reach 0.8 sigma past a cell's faces,
    and a replica with a site beyond runs in FP64.  40 sigma stands for a
    state that blows up."""
    s = C.config_droplet(240, 4, cells=(8, 8, 8), seed=12)
    pos = s.pos.copy()
    pos[:3 * s.n_water].reshape(-1, 9)[::3, ::3] += drift
    o, eng = O.Oracle(s), E.Engine(s, precision)
    o.force(True, terms=E.T_NEAR)
    eng.force(True, terms=E.T_NEAR)
    o.set(0, pos)
    eng.set_state(pos)
    fo = o.force(False, terms=E.T_NEAR)
    assert rel(eng.force(False, terms=E.T_NEAR), fo) < bar


@pytest.mark.parametrize("r", [0.3, 0.35, 0.36, 0.5, 1.0, 2.0, 4.0, 5.25])
def test_plain_pair_at_exact_distances(r):
    """Two waters whose oxygens are r sigma apart along an axis: powers of two,
    where the scaled distance of the FP64 path's integers meets the ends of
    its range, and both sides of the distance below which it uses FP64."""
    s = grid_waters(2, 3.0, seed=1)
    wt = S.water_template() / S.SIGMA
    pos = np.concatenate([wt, -wt]) + 0.25
    pos[3:, 0] += r
    s = dataclasses.replace(s, pos=pos)
    fo = O.Oracle(s).force(True, terms=E.T_NEAR)
    assert rel(E.Engine(s, E.PLAIN_FP64).force(True, terms=E.T_NEAR), fo) < 1e-13
