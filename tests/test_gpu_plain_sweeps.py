"""Both halves of the plain path against the reference's Gauss-Seidel sweeps
(src/move_w1_a.f90:36-134, src/move_w1_b.f90:30-119 and the surfactants'
src/move_surfactant_a.f90, src/move_surfactant_b.f90), restated here in NumPy
one rounding an operation, with any limit of sweeps: the same bits and the
same molecules counted as failed."""
import ctypes

import numpy as np
import pytest

import oracle as O
from surfactant_enhanced_spreading_gb300 import engine as E
from surfactant_enhanced_spreading_gb300 import system as S

TOL = 1e-4


def _constants():
    lib = O.lib()
    c, ds, bonds = np.empty(8), np.empty(28), np.empty(56, dtype=np.int32)
    lib.orc_constants(O._dp(c))
    lib.orc_table_dsqs.argtypes = [ctypes.POINTER(ctypes.c_double)]
    lib.orc_table_dsqs(O._dp(ds))
    lib.orc_table_bonds.argtypes = [ctypes.POINTER(ctypes.c_int)]
    lib.orc_table_bonds(bonds.ctypes.data_as(ctypes.POINTER(ctypes.c_int)))
    water = ([(0, 1), (1, 2), (2, 0)], np.array([c[6], c[7], c[6]]))
    return c[5], water, ([tuple(b) for b in bonds.reshape(28, 2) - 1], ds)


def dot(a, b):
    return a[:, 0] * b[:, 0] + a[:, 1] * b[:, 1] + a[:, 2] * b[:, 2]


def species(s):
    """(first site, sites of a molecule, bonds, squared lengths) of the waters and of the surfactants."""
    dt, water, surf = _constants()
    n = 3 * s.n_water
    return dt, [(slice(0, n), 3, *water), (slice(n, s.n_sites), 29, *surf)]


def sweeps(bonds, maxit, n, act):
    """act(bond number, molecules) -> which of them it corrected.  Molecules that ran out of sweeps."""
    active = np.arange(n)
    for _ in range(maxit + 1):
        changed = np.zeros(n, dtype=bool)
        for b in range(len(bonds)):
            changed[active] |= act(b, active)
        active = active[changed[active]]
    return len(active)


def shake(s, pos, vel, acc, eta, maxit):
    dt, kinds = species(s)
    escale = 1.0 - eta * dt / 2.0
    p, v, fails, mass = pos + vel * escale + acc, vel * escale + acc, 0, s.masses()
    for sl, ns, bonds, dsq in kinds:
        P, V, R = p[sl].reshape(-1, ns, 3), v[sl].reshape(-1, ns, 3), pos[sl].reshape(-1, ns, 3)
        im = 1.0 / mass[sl][:ns]

        def act(b, m):
            i, j = bonds[b]
            pab, rab = P[m, i] - P[m, j], R[m, i] - R[m, j]
            diff = dsq[b] - dot(pab, pab)
            cor = np.abs(diff) > dsq[b] * (2.0 * TOL)
            c = m[cor]
            d = rab[cor] * (diff / (2.0 * (im[i] + im[j]) * dot(rab, pab)))[cor, None]
            P[c, i] += im[i] * d; P[c, j] -= im[j] * d
            V[c, i] += im[i] * d; V[c, j] -= im[j] * d
            return cor

        if len(P):
            fails += sweeps(bonds, maxit, len(P), act)
    return p, v, fails


def rattle(s, pos, vel, force, eta, maxit):
    dt, kinds = species(s)
    mass = s.masses()
    acc = force * (dt * dt / 2.0) / mass[:, None]
    v, fails = 2.0 / (2.0 + eta * dt) * (vel + acc), 0
    for sl, ns, bonds, dsq in kinds:
        V, R = v[sl].reshape(-1, ns, 3), pos[sl].reshape(-1, ns, 3)
        im = 1.0 / mass[sl][:ns]

        def act(b, m):
            i, j = bonds[b]
            vab, rab = V[m, i] - V[m, j], R[m, i] - R[m, j]
            gab = -(dot(rab, vab) / dt) / ((im[i] + im[j]) * dsq[b])
            cor = np.abs(gab) > TOL
            c = m[cor]
            d = rab[cor] * gab[cor, None]
            V[c, i] += im[i] * d * dt
            V[c, j] -= im[j] * d * dt
            return cor

        if len(V):
            fails += sweeps(bonds, maxit, len(V), act)
    return acc, v, fails


def state(water, surf):
    s = S.droplet(water, surf, cells=(8, 8, 4) if water < 1000 else (16, 16, 8), seed=water + surf)
    return s, np.random.default_rng(7).normal(size=s.pos.shape) * (1e-4 / s.masses())[:, None]


def test_restatement_equals_the_oracle():
    s, acc = state(31, 4)
    o = O.Oracle(s)
    o.set(2, acc)
    o.move_a()
    p, v, fails = shake(s, s.pos, s.vel, acc, 0.0, 100)
    assert np.array_equal(p, o.get(0)) and np.array_equal(v, o.get(1)) and fails == o.fail_count()
    o = O.Oracle(s)
    f = o.force(True)
    o.eta = 0.3
    o.move_b()
    a, v, fails = rattle(s, s.pos, s.vel, f, 0.3, 100)
    assert np.array_equal(a, o.get(2)) and np.array_equal(v, o.get(1)) and fails == o.fail_count()


# the last group of 10 waters part filled; one lane a water above 6,080 waters
@pytest.mark.gpu
@pytest.mark.parametrize("water,surf", [(1, 0), (9, 1), (10, 2), (11, 3), (31, 4), (200, 7), (6080, 1), (6081, 1)])
@pytest.mark.parametrize("maxit", [100, 5, 3, 1, 0, -1])
def test_halves_equal_the_sweeps(water, surf, maxit):
    s, acc = state(water, surf)
    eng = E.Engine(s, E.PLAIN_FP64, shake_maxit=maxit)
    eng.set_state(s.pos, s.vel, acc, 0.3)
    eng.move_a()
    p, v, fails = shake(s, s.pos, s.vel, acc, 0.3, maxit)
    pos, vel, _ = eng.state()
    assert np.array_equal(pos, p) and np.array_equal(vel, v)
    assert eng.failures()[0] == fails
    for terms in (0, E.T_ALL):
        before = eng.failures()[0]
        eng.set_state(s.pos, s.vel, acc, 0.3)
        f = eng.force(True, terms=terms)
        eng.move_b()
        a, v, fails = rattle(s, s.pos, s.vel, f, 0.3, maxit)
        _, vel, out = eng.state()
        assert np.array_equal(out, a) and np.array_equal(vel, v)
        assert eng.failures()[0] - before == fails
