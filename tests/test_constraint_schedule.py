"""The surfactants' wavefronts (a bond at a fixed step of its sweep, sweeps 4 or
6 steps apart) restated on the CPU: every schedule gives the bits, the sweep
count and the verdict of the sequential Gauss-Seidel sweeps."""
import numpy as np
import pytest

from surfactant_enhanced_spreading_gb300 import system as S

BONDS = 28
END = 23


def place(b):
    return b if b <= 22 else b - 4 if b <= 26 else END


class Molecule:
    """SHAKE over the bonds of one surfactant, plain FP64 (one rounding an operation)."""

    def __init__(self, seed):
        rng = np.random.default_rng(seed)
        self.b = TOPOLOGY
        self.r = START + rng.normal(size=START.shape) * 1e-3
        self.p = self.r + rng.normal(size=START.shape) * 2e-2
        self.d2 = np.array([((START[i] - START[j]) ** 2).sum() for i, j in self.b])
        self.im = 1.0 / MASS

    def act(self, b, tol):
        i, j = self.b[b]
        p, r = self.p[i] - self.p[j], self.r[i] - self.r[j]
        diff = self.d2[b] - ((p[0] * p[0] + p[1] * p[1]) + p[2] * p[2])
        if not abs(diff) > self.d2[b] * (2.0 * tol):
            return False
        g = diff / (2.0 * (self.im[i] + self.im[j]) * ((r[0] * p[0] + r[1] * p[1]) + r[2] * p[2]))
        self.p[i] = self.p[i] + self.im[i] * (r * g)
        self.p[j] = self.p[j] - self.im[j] * (r * g)
        return True


def sequential(m, tol, maxit):
    for _ in range(maxit + 1):
        if not any([m.act(b, tol) for b in range(BONDS)]):
            return True
    return False


def wavefront(m, tol, maxit, lag):
    """The kernel's rule: lines of sweeps, a branch line, flags kept a step."""
    lines = (END + 1) // lag
    assert lines * lag == END + 1
    if maxit < 0:
        return False
    sweep = list(range(lines)) + [0]
    dirty = [False] * (lines + 1)
    branch_dirty = False
    step = 0
    while True:
        ended = []
        for u in range(lines + 1):
            branch = u == lines
            tau = step - lag * sweep[u]
            on = sweep[u] <= maxit and ((19 <= tau <= 22) if branch else tau >= 0)
            if on:
                b = tau + 4 if branch else BONDS - 1 if tau == END else tau
                dirty[u] = m.act(b, tol) or dirty[u]
                if not branch and tau == END:
                    ended.append(u)
        clean = any(not dirty[u] and not branch_dirty for u in ended)
        out = any(sweep[u] == maxit for u in ended)
        for u in ended:
            dirty[u] = False
            sweep[u] += lines
        if step - lag * sweep[lines] == 22:
            branch_dirty, dirty[lines] = dirty[lines], False
            sweep[lines] += 1
        if clean:
            return True
        if out:
            return False
        step += 1


def _start():
    s = S.droplet(20, 1, cells=(8, 8, 4), seed=1)
    return s.pos[3 * s.n_water:].copy(), s.masses()[3 * s.n_water:].copy()


START, MASS = _start()
TOPOLOGY = [(i - 1, j - 1) for i, j in S.SURF_BONDS]


@pytest.mark.parametrize("lag", [4, 6, 8])
def test_bonds_that_share_a_site_keep_their_order(lag):
    """Within a sweep the later bond comes later, and before the next sweep's earlier one."""
    for a in range(BONDS):
        for b in range(a + 1, BONDS):
            if set(TOPOLOGY[a]) & set(TOPOLOGY[b]):
                assert 1 <= place(b) - place(a) < lag


@pytest.mark.parametrize("lag", [4, 6])
@pytest.mark.parametrize("tol,maxit", [(1e-4, 100), (1e-8, 100), (1e-4, 3), (1e-8, 5), (1e-4, 1), (1e-4, 0), (10.0, 100), (1e-4, -1)])
def test_wavefront_equals_the_sweeps(lag, tol, maxit):
    for seed in range(3):
        a, b = Molecule(seed), Molecule(seed)
        assert sequential(a, tol, maxit) == wavefront(b, tol, maxit, lag)
        assert np.array_equal(a.p, b.p)
