"""Performance cases: the work a user has the engine do, through its Python binding.

A case is one droplet (or a batch of droplets) in one precision mode, and one
of four call sequences on a kept engine:

* ``run``: a stretch of a spreading run: state in (``set_state``), start-up
  force and accelerations (``mybox_start``), 19 steps (``run``) and the state
  out.  20 force calls, 2 of them with the
  lists and the far field rebuilt: the engine's 1-in-10 schedule;
* ``loop``: the same driven step by step as a Fortran host drives it
  (``step`` and ``temperature`` every step);
* ``halves``: one step through the drop-in calls (``move_a``, ``force``,
  ``move_b``) from a state that the host holds, with a rebuild, and one from
  the next state with frozen lists.  The reference preset's mixed paths are
  measured so: their sweeps stop anywhere inside a 1e-4 tolerance, so over
  several steps two roundings of one force part by that much;
* ``force``: the force section alone, once with a rebuild and once with frozen
  lists at positions one step later, as a host with its own integrator
  calls it.

The state is host data by the interface's nature, so ``prepare`` keeps it
there.  Droplets come from the repository's own generators; a seed turns and
shifts the droplet and draws new velocities.  The mixed paths compute their
forces in FP32, so their program keeps its frames in FP32, as a trajectory
is stored; the plain path's outputs stay in FP64.

``exact`` restates the configuration preset in FP64 torch: near field over the
27 cells, order-4 multipole far field, chain terms, graphite, walls, exact
solutions of the water constraints, Nose-Hoover.  The reference preset's
states have no such value (the 1e-4 tolerance again).
"""
import dataclasses
import functools
import itertools
import math

import numpy as np
import torch

from surfactant_enhanced_spreading_gb300 import config_preset as C
from surfactant_enhanced_spreading_gb300 import engine as E
from surfactant_enhanced_spreading_gb300 import serve
from surfactant_enhanced_spreading_gb300 import system as S

MODES = {"plain": E.PLAIN_FP64, "mixed": E.MIXED, "fp32c": E.MIXED_FP32C, "comp": E.MIXED_COMP}
KB0, STEPS = 99101, 19      # one rebuild step (99110) beside the start-up's


def listed():
    def case(name, kind, preset, mode, water, surf, cells="", layers=2, replicas=1):
        return dict(name=name, kind=kind, preset=preset, mode=mode, water=water, surf=surf, cells=cells,
                    layers=layers, replicas=replicas)
    return [
        # the small configuration, on both paths: latency and launches count
        case("small_run", "run", "config", "mixed", 1000, 0, "8,8,8"),
        case("small_plain_run", "run", "config", "plain", 1000, 0, "8,8,8"),
        # the medium configuration: its steps, and the FP64 force section its results are checked with
        case("medium_run", "run", "config", "mixed", 20000, 200, "20,20,12", 4),
        case("medium_plain_force", "force", "config", "plain", 20000, 200, "20,20,12", 4),
        # the large configuration, the benchmark's headline
        case("large_run", "run", "config", "mixed", 100000, 1000, "40,40,16", 4),
        # an ensemble of uneven replicas advanced by every launch, sized as the batched configuration draws them
        case("ensemble_run", "run", "config", "mixed", 30000, 600, "", 2, 8),
        # a served request's size, driven step by step by a host that reads the temperature
        case("served_loop", "loop", "config", "mixed", 7003, 35),
        # compensated sums: the option for the smallest force error
        case("compensated_force", "force", "config", "comp", 13331, 133),
        # the reference's force field: its benchmark droplet, a surfactant-rich one, FP32 constraints, the FP64 path
        case("reference_halves", "halves", "reference", "mixed", 20000, 200, "24,24,12"),
        case("surfactant_halves", "halves", "reference", "mixed", 3001, 120, "16,16,8"),
        case("fp32c_halves", "halves", "reference", "fp32c", 5000, 50, "16,16,8"),
        case("reference_plain_run", "run", "reference", "plain", 701, 12, "8,8,8"),
    ]


def draw(rng):
    """A droplet of 300 to 60,000 waters (fewer on the plain path) with up to 2 % chains or surfactants."""
    def logu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    preset = rng.choice(["config", "config", "config", "reference"])
    mode = rng.choice(["mixed", "mixed", "mixed", "comp", "plain"] + ["fp32c"] * (preset == "reference"))
    kind = rng.choice(["run", "run", "loop", "halves", "force"])
    if preset == "reference" and mode != "plain":
        kind = rng.choice(["halves", "force"])
    replicas = rng.choice([1, 1, 1, 3, 5]) if preset == "config" and kind == "run" and mode != "plain" else 1
    top = {"config": 60000, "reference": 20000}[preset] if mode != "plain" else (20000 if kind == "force" else 2500)
    water = logu(300, top // (1 if replicas == 1 else 4))
    surf = int(round(water * rng.uniform(0.0, 0.02 if preset == "config" else 0.01)))
    return dict(kind=kind, preset=preset, mode=mode, water=water, surf=surf, cells="", layers=rng.choice([2, 4]),
                replicas=replicas)


# ---------------------------------------------------------------- inputs

@functools.lru_cache(maxsize=None)
def _droplet(preset, water, surf, cells, layers):
    if preset == "config":
        if not cells:
            n = C.sheet_cells(water)
            cells = (n, n, C.box_height_cells(water, surf))
        return C.config_droplet(water, surf, cells=cells, seed=2024, graphite_layers=layers)
    if not cells:
        return serve.make_request(0, water, surf, 1, seed=2024).system
    return S.droplet(water, surf, cells=cells, seed=2024, graphite_layers=layers)


def _bases(case):
    """The case's droplets: one, or replicas from its size down to 1/30 of it in even ratios."""
    cells = tuple(int(c) for c in case["cells"].split(",")) if case["cells"] else None
    n = case["replicas"]
    out = []
    for k in range(n):
        f = 30.0 ** (-k / (n - 1)) if n > 1 else 1.0
        out.append(_droplet(case["preset"], max(100, round(case["water"] * f)), round(case["surf"] * f), cells,
                            case["layers"]))
    return out


def _velocities(s, pos, rng):
    """Maxwell velocities at the preset's temperature; the waters' part along their rigid bonds is taken out."""
    mass = s.masses()
    v = rng.normal(size=(mass.size, 3)) * np.sqrt((C.TR if s.preset else S.TR) / mass)[:, None]
    nw = 3 * s.n_water
    w, p, im = v[:nw].reshape(-1, 3, 3), pos[:nw].reshape(-1, 3, 3), 1.0 / S.WATER_MASS
    bonds = [(0, 1), (1, 2), (2, 0)]
    r = np.stack([p[:, i] - p[:, j] for i, j in bonds], 1)
    sign = np.array([[(1.0 if k == i else -1.0 if k == j else 0.0) for k in range(3)] for i, j in bonds])
    a = np.einsum("ak,bk,k->ab", sign, sign, im)[None] * np.einsum("nax,nbx->nab", r, r)
    g = np.linalg.solve(a, np.einsum("ak,nkx,nax->na", sign, w, r)[..., None])[..., 0]
    v[:nw] = (w - np.einsum("bk,k,nb,nbx->nkx", sign, im, g, r)).reshape(-1, 3)
    return v * S.DT


def _systems(case, seed):
    """The droplets turned by quarter turns about z, mirrored, shifted (anywhere in a periodic box, by up to
    0.5 A in a closed one) and given new velocities."""
    out = []
    for k, s in enumerate(_bases(case)):
        rng = np.random.default_rng([seed, k])
        pos = s.pos.copy()
        if s.cells[0] == s.cells[1] and rng.integers(2):
            pos[:, [0, 1]] = pos[:, [1, 0]]
        pos[:, :2] *= rng.choice([-1.0, 1.0], 2)
        span = s.half_box[:2] if s.preset else 0.5 / S.SIGMA
        pos[:, :2] += rng.uniform(-1.0, 1.0, 2) * span
        out.append(dataclasses.replace(s, pos=pos, vel=_velocities(s, pos, rng)))
    return out


def _accelerations(case, systems, seed):
    """A run computes its own at the start; the halves get some of the usual size."""
    acc = np.zeros((sum(s.n_sites for s in systems), 3))
    if case["kind"] == "halves":
        mass = np.concatenate([s.masses() for s in systems])
        acc += np.random.default_rng([seed, 99]).normal(size=acc.shape) * (1e-4 / mass)[:, None]
    return acc


def prepare(case, seed):
    systems = _systems(case, seed)
    pos = np.concatenate([s.pos for s in systems])
    vel = np.concatenate([s.vel for s in systems])
    eng = E.Engine(systems if len(systems) > 1 else systems[0], MODES[case["mode"]])
    return dict(eng=eng, kind=case["kind"], fp32=case["mode"] != "plain", pos=pos, vel=vel, pos1=pos + vel,
                acc=_accelerations(case, systems, seed), out=tuple(np.empty_like(pos) for _ in range(3)))


def _frame(state, *arrays):
    return [torch.from_numpy(a).float() if state["fp32"] else torch.from_numpy(a.copy()) for a in arrays]


def run(state):
    eng = state["eng"]
    if state["kind"] == "force":
        eng.set_state(state["pos"])
        f0 = eng.force(True)
        eng.set_state(state["pos1"])
        return _frame(state, f0, eng.force(False))
    if state["kind"] == "halves":
        out = []
        for pos, rebuild in ((state["pos"], True), (state["pos1"], False)):
            eng.set_state(pos, state["vel"], state["acc"], 0.0)
            eng.move_a()
            f = eng.force(rebuild)
            eng.move_b()
            eng.state(out=state["out"])
            out += _frame(state, f, *state["out"], eng.etas())
        return out
    eng.set_state(state["pos"], state["vel"], state["acc"], 0.0)
    E.mybox_start(eng)
    if state["kind"] == "loop":
        temps = np.empty(STEPS)
        for k in range(STEPS):
            eng.step(KB0 + k)
            temps[k] = eng.temperature()
        eng.state(out=state["out"])
        return _frame(state, *state["out"], temps)
    eng.run(KB0, STEPS)
    eng.state(out=state["out"])
    return _frame(state, *state["out"], eng.etas())


def work(case):
    """Bytes: the state in and the forces and state out.  Operations of the near field (18 a site pair), the
    local expansion (1,000 a site) and the integrator (300 a site and step)."""
    pairs = sites = 0.0
    for k in range(case["replicas"]):
        f = 30.0 ** (-k / (case["replicas"] - 1)) if case["replicas"] > 1 else 1.0
        nw, ns = max(100, round(case["water"] * f)), round(case["surf"] * f)
        n = 3 * nw + (12 if case["preset"] == "config" else 29) * ns
        # share of a 36 A cube about a site of a half ball that lies inside it
        rng = np.random.default_rng(0)
        radius = (3.0 * n / (2.0 * math.pi * 0.1002)) ** (1.0 / 3.0)
        p = rng.uniform(-1, 1, (4000, 3)) * radius
        p[:, 2] = np.abs(p[:, 2])
        p = p[(p ** 2).sum(1) < radius ** 2]
        q = p + rng.uniform(-18.0, 18.0, p.shape)
        inside = ((q ** 2).sum(1) < radius ** 2) & (q[:, 2] > 0)
        pairs += n * 0.1002 * 36.0 ** 3 * float(inside.mean())
        sites += n
    evals, moves = {"force": (2, 0), "halves": (2, 2)}.get(case["kind"], (STEPS + 1, STEPS))
    flops = evals * (18.0 * pairs + 1000.0 * sites) + moves * 300.0 * sites
    per_site = {"force": 2 * (24 + 24), "halves": 2 * (72 + 96)}.get(case["kind"], 72 + 24 + 72)
    return {"bytes": per_site * sites, "flops": flops}


# ---------------------------------------------------------------- the same in 64 bits

ORDER = 4
KJ = 1000.0 / 650.2                      # kJ/mol in the reduced energy
XPI = float(np.float32(675.05))          # Coulomb prefactor
BEADS = 12
CHARGE = [-0.82, 0.41, 0.40, -0.60, 0.60, -0.40] + [0.0] * 8
MASS = [1.0, 1.00794 / 15.9994] + [m / 15.9994 for m in [15.035, 15.9994, 14.027, 15.9994] + [14.027] * 8]
LJ_SIGMA = [x / 3.166 for x in [3.166, 0.0, 3.75, 2.80, 3.95, 2.80] + [3.9] * 8]
LJ_EPS = [x * KJ for x in [0.65, 0.0, 0.815, 0.457, 0.382, 0.457] + [0.38] * 8]
NM = [(n, m) for n in range(2 * ORDER + 1) for m in range(-n, n + 1)]
AT = {nm: k for k, nm in enumerate(NM)}
LOW = (ORDER + 1) ** 2


def _regular(r, order):
    """r^n P_n^m e^(i m phi) / (n + m)!, all m, as (..., (order + 1)^2) complex values."""
    x, y, z = r.unbind(-1)
    xy, r2 = torch.complex(x, y), (r * r).sum(-1)
    t = {(0, 0): torch.ones_like(xy)}
    for n in range(1, order + 1):
        t[n, n] = t[n - 1, n - 1] * xy / (-2.0 * n)
        for m in range(n):
            low = t[n - 2, m] * r2 if (n - 2, m) in t else 0.0
            t[n, m] = ((2 * n - 1) * z * t[n - 1, m] - low) / ((n + m) * (n - m))
    return torch.stack([t[n, m] if m >= 0 else (-1) ** m * t[n, -m].conj() for n, m in NM[:(order + 1) ** 2]], -1)


def _irregular(r, order):
    """(n - m)! P_n^m e^(i m phi) / r^(n + 1), all m."""
    x, y, z = r.unbind(-1)
    xy, r2 = torch.complex(x, y), (r * r).sum(-1)
    t = {(0, 0): (1.0 / r2.sqrt()).to(xy.dtype)}
    for n in range(1, order + 1):
        t[n, n] = -(2 * n - 1) * xy / r2 * t[n - 1, n - 1]
        for m in range(n):
            low = ((n - 1) ** 2 - m * m) * t[n - 2, m] if (n - 2, m) in t else 0.0
            t[n, m] = ((2 * n - 1) * z * t[n - 1, m] - low) / r2
    return torch.stack([t[n, m] if m >= 0 else (-1) ** m * t[n, -m].conj() for n, m in NM[:(order + 1) ** 2]], -1)


def _m2l(irr):
    """Multipole-to-local operators (..., out, in) of order 4 from the irregular harmonics of target - source."""
    idx = torch.tensor([[AT[n + j, m + k] for n, m in NM[:LOW]] for j, k in NM[:LOW]], device=irr.device)
    sign = torch.tensor([(-1.0) ** j for j, _ in NM[:LOW]], device=irr.device, dtype=torch.float64)
    return irr[..., idx] * sign[:, None]


class _Exact:
    """The configuration preset of one droplet."""

    def __init__(self, s):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        f64 = functools.partial(torch.tensor, dtype=torch.float64, device=self.dev)
        self.nw, self.ns, self.nc = s.n_water, s.n_surf, s.cells
        self.box = f64([c * S.RS for c in s.cells])
        self.half = self.box / 2
        self.x, self.v, self.a, self.eta = f64(s.pos), f64(s.vel), torch.zeros_like(f64(s.pos)), 0.0
        n = s.n_sites
        kind = np.concatenate([np.tile([0, 1, 1], s.n_water), np.tile(np.arange(2, 14), s.n_surf)]).astype(np.int64)
        mol = np.concatenate([np.arange(3 * s.n_water) // 3, s.n_water + np.arange(BEADS * s.n_surf) // BEADS])
        self.kind, self.mol = torch.tensor(kind, device=self.dev), torch.tensor(mol.astype(np.int64), device=self.dev)
        self.q, self.m = f64(CHARGE)[self.kind], f64(MASS)[self.kind]
        sg, ep = f64(LJ_SIGMA), f64(LJ_EPS)
        on = (sg > 0).double()
        s6 = ((sg[:, None] + sg) / 2) ** 6
        self.s6, self.e48 = s6, 48.0 * (ep[:, None] * ep).sqrt() * s6 * on[:, None] * on
        self.gs6 = ((sg + 3.4 / 3.166) / 2) ** 6
        self.ge48 = 48.0 * (ep * 0.23 * KJ).sqrt() * self.gs6 * on
        self.carb = f64(s.carbons.reshape(-1, 3)) if s.graphite_on else None
        if self.carb is not None and len(self.carb):
            self.igz = int(min(max(math.floor(float((self.carb[:, 2].max() + S.RS + self.half[2]) / S.RS)), 0), self.nc[2] - 1))
            col = torch.floor((self.carb[:, :2] + self.half[:2]) / S.RS).long()
            col = torch.stack([col[:, a] % self.nc[a] for a in (0, 1)], 1)
            self.ctab = self._table(col[:, 0] + self.nc[0] * col[:, 1], self.nc[0] * self.nc[1])
        else:
            self.carb = None
        self.dof = 3 * n - 3 * s.n_water
        rlx = C.TAU_STEPS * S.DT
        self.pnh1, self.pnh2 = S.DT / self.dof / C.TR / rlx ** 2, -2.0 * self.dof * C.TR

    def _table(self, cell, ncell):
        """Members of each cell, padded with -1."""
        count = torch.bincount(cell, minlength=ncell)
        order = torch.argsort(cell, stable=True)
        rank = torch.arange(len(cell), device=self.dev) - (torch.cumsum(count, 0) - count)[cell[order]]
        t = torch.full((ncell, int(count.max())), -1, dtype=torch.long, device=self.dev)
        t[cell[order], rank] = order
        return t

    def _centre(self, idx, size):
        return -self.half + (idx.double() + 0.5) * size

    # lists and local expansions, frozen until the next rebuild
    def rebuild(self):
        nx, ny, nz = self.nc
        self.ext = torch.floor((self.x + self.half) / S.RS).long()
        image = torch.stack([torch.div(self.ext[:, 0], nx, rounding_mode="floor"),
                             torch.div(self.ext[:, 1], ny, rounding_mode="floor"),
                             torch.zeros_like(self.ext[:, 2])], 1)
        self.shift = image.double() * self.box
        self.cxyz = self.ext - image * torch.tensor(self.nc, device=self.dev)
        assert bool(((self.cxyz[:, 2] >= 0) & (self.cxyz[:, 2] < nz)).all())
        self.cell = self.cxyz[:, 0] + nx * (self.cxyz[:, 1] + ny * self.cxyz[:, 2])
        self.table = self._table(self.cell, nx * ny * nz)
        w = self.x - self.shift
        self.local = []
        for size in (1, 2, 4):
            n = [c // size for c in self.nc]
            b = self.cxyz // size
            flat = b[:, 0] + n[0] * (b[:, 1] + n[1] * b[:, 2])
            mom = torch.zeros(n[0] * n[1] * n[2], LOW, dtype=torch.complex128, device=self.dev)
            mom.index_add_(0, flat, _regular(w - self._centre(b, size * S.RS), ORDER).conj() * self.q[:, None])
            mom = mom.view(n[2], n[1], n[0], LOW)
            loc = self._top(mom, n) if size == 4 else self._lists(mom, n, size * S.RS)
            self.local.append((size, b, loc.reshape(-1, LOW)[flat]))

    def _lists(self, mom, n, size):
        """Children of the parent's neighbours that are not neighbours, per parity of the target."""
        out = torch.zeros_like(mom)
        offs = torch.tensor(list(itertools.product(range(-3, 4), repeat=3)), device=self.dev)      # source - target
        ops = torch.zeros(343, LOW, LOW, dtype=mom.dtype, device=self.dev)
        far = offs.abs().amax(1) > 1
        ops[far] = _m2l(_irregular(-offs[far].double() * size, 2 * ORDER))
        padded = torch.zeros(n[2] + 6, n[1], n[0], LOW, dtype=mom.dtype, device=self.dev)
        padded[3:-3] = mom
        for dx, dy, dz in itertools.product(range(-3, 4), repeat=3):
            if max(abs(dx), abs(dy), abs(dz)) <= 1:
                continue
            # parity p of a target's index admits offsets -2 - p .. 3 - p
            px, py, pz = ([p for p in (0, 1) if -2 - p <= o <= 3 - p] for o in (dx, dy, dz))
            src = torch.roll(padded[3 + dz:3 + dz + n[2]], (-dy, -dx), (1, 2))
            for a, b, c in itertools.product(px, py, pz):
                out[c::2, b::2, a::2] += src[c::2, b::2, a::2] @ ops[(dx + 3) * 49 + (dy + 3) * 7 + dz + 3].T
        return out

    def _top(self, mom, n):
        """Every box and image of the 3 x 3 supercell that is not a neighbour."""
        spans = [torch.arange(-(k - 1), k, device=self.dev) for k in n]
        off = torch.cartesian_prod(*spans)                      # source - target
        fac = torch.zeros(len(off), len(NM), dtype=mom.dtype, device=self.dev)
        for ix, iy in itertools.product((-1, 0, 1), repeat=2):
            o = off + torch.tensor([ix * n[0], iy * n[1], 0], device=self.dev)
            far = o.abs().amax(1) > 1
            fac[far] += _irregular(-o[far].double() * 4 * S.RS, 2 * ORDER)
        box = torch.cartesian_prod(*[torch.arange(k, device=self.dev) for k in (n[2], n[1], n[0])]).flip(1)
        flat = mom.reshape(-1, LOW)
        out = torch.empty_like(flat)
        for k in range(len(box)):
            d = box - box[k] + torch.tensor([c - 1 for c in n], device=self.dev)
            op = _m2l(fac[(d[:, 0] * (2 * n[1] - 1) + d[:, 1]) * (2 * n[2] - 1) + d[:, 2]])
            out[k] = torch.einsum("sab,sb->a", op, flat)
        return out

    def force(self):
        f = self._near() + self._far()
        if self.ns:
            f[3 * self.nw:] += self._chains()
        up, down = self.x[:, 2] - self.half[2], self.half[2] + self.x[:, 2]
        f[:, 2] += 48.0 / up ** 13 + 48.0 / down ** 13
        if self.carb is not None:
            self._graphite(f)
        return f

    def _near(self):
        nx, ny, nz = self.nc
        w = self.x - self.shift
        f = torch.zeros_like(self.x)
        full = torch.nonzero(self.table[:, 0] >= 0)[:, 0]
        m = self.table.shape[1]
        step = max(1, (1 << 24) // (m * m))
        flat_e, flat_s = self.e48.reshape(-1), self.s6.reshape(-1)
        for c0 in range(0, len(full), step):
            c = full[c0:c0 + step]
            xyz = torch.stack([c % nx, (c // nx) % ny, c // (nx * ny)], 1)
            ti = self.table[c]
            live_i = ti >= 0
            pi, ki, mi = w[ti], self.kind[ti], self.mol[ti]
            acc = torch.zeros_like(pi)
            for dz, dy, dx in itertools.product((-1, 0, 1), repeat=3):
                o = xyz + torch.tensor([dx, dy, dz], device=self.dev)
                inside = (o[:, 2] >= 0) & (o[:, 2] < nz)
                wrapped = torch.stack([o[:, 0] % nx, o[:, 1] % ny, o[:, 2].clamp(0, nz - 1)], 1)
                shift = (o - wrapped).double() * S.RS * torch.tensor([1.0, 1.0, 0.0], device=self.dev)
                tj = self.table[wrapped[:, 0] + nx * (wrapped[:, 1] + ny * wrapped[:, 2])]
                live = live_i[:, :, None] & (tj >= 0)[:, None] & inside[:, None, None] & (mi[:, :, None] != self.mol[tj][:, None])
                d = pi[:, :, None] - (w[tj] + shift[:, None])[:, None]
                r2 = torch.where(live, (d * d).sum(-1), 1.0)
                i2 = 1.0 / r2
                g = (self.q[ti] * XPI)[:, :, None] * self.q[tj][:, None] * i2 * i2.sqrt()
                pair = ki[:, :, None] * len(CHARGE) + self.kind[tj][:, None]
                i6 = i2 * i2 * i2
                g = g + torch.where(r2 <= S.RC ** 2, flat_e[pair] * i6 * (flat_s[pair] * i6 - 0.5) * i2, 0.0)
                acc += (d * torch.where(live, g, 0.0)[..., None]).sum(2)
            f[ti[live_i]] = acc[live_i]
        return f

    def _far(self):
        """Gradient of sum L_n^m conj(R_n^m): d/dz R_n^m = R_(n-1)^m, (d/dx +- i d/dy) R_n^m = +-R_(n-1)^(m +- 1)."""
        grad = torch.zeros_like(self.x)
        w = self.x - self.shift
        for size, b, loc in self.local:
            reg = _regular(w - self._centre(b, size * S.RS), ORDER - 1)
            for n, m in NM[1:LOW]:
                get = lambda k: reg[:, AT[n - 1, k]] if abs(k) <= n - 1 else 0.0  # noqa: E731
                plus, minus = get(m + 1), -get(m - 1)
                coef = loc[:, AT[n, m]]
                for a, d in enumerate(((plus + minus) / 2, (plus - minus) / 2j, get(m))):
                    grad[:, a] += (coef * d.conj()).real if torch.is_tensor(d) else 0.0
        return -grad * (self.q * XPI)[:, None]

    def _chains(self):
        r = self.x[3 * self.nw:].view(-1, BEADS, 3).detach().clone().requires_grad_(True)
        bond = r[:, :-1] - r[:, 1:]
        ln = bond.norm(dim=-1)
        u = (1000.0 * KJ * 3.166 ** 2 * (ln - 1.53 / 3.166) ** 2).sum()
        cos = -(bond[:, :-1] * bond[:, 1:]).sum(-1) / (ln[:, :-1] * ln[:, 1:])
        u = u + (0.5 * 519.7 * KJ * (torch.acos(cos) - math.radians(112.0)) ** 2).sum()
        m, n = torch.linalg.cross(bond[:, :-2], bond[:, 1:-1]), torch.linalg.cross(bond[:, 1:-1], bond[:, 2:])
        c = (m * n).sum(-1) / (m.norm(dim=-1) * n.norm(dim=-1))
        u = u + (KJ * (2.9517 * (1 + c) - 0.5669 * (1 - (2 * c * c - 1)) + 6.5790 * (1 + 4 * c ** 3 - 3 * c))).sum()
        i, j = torch.triu_indices(BEADS, BEADS, 4, device=self.dev)
        k = torch.arange(2, 2 + BEADS, device=self.dev)
        qq = torch.tensor(CHARGE, dtype=torch.float64, device=self.dev)[k]
        r2 = ((r[:, i] - r[:, j]) ** 2).sum(-1)
        i6 = 1.0 / r2 ** 3
        u = u + (XPI * qq[i] * qq[j] / r2.sqrt() + self.e48[k[i], k[j]] / 12 * (self.s6[k[i], k[j]] * i6 * i6 - i6)).sum()
        i, j = torch.triu_indices(BEADS, BEADS, 1, device=self.dev)
        e = self.ext[3 * self.nw:].view(-1, BEADS, 3)
        apart = (e[:, i] - e[:, j]).abs().amax(-1) > 1
        r2 = torch.where(apart, ((r[:, i] - r[:, j]) ** 2).sum(-1), 1.0)
        u = u - torch.where(apart, XPI * qq[i] * qq[j] / r2.sqrt(), 0.0).sum()
        return -torch.autograd.grad(u, r)[0].reshape(-1, 3)

    def _graphite(self, f):
        site = torch.nonzero((self.cxyz[:, 2] <= self.igz) & (self.ge48[self.kind] > 0))[:, 0]
        step = max(1, (1 << 24) // self.ctab.shape[1])
        nx, ny, _ = self.nc
        for s0 in range(0, len(site), step):
            s = site[s0:s0 + step]
            p, e48, s6 = (self.x - self.shift)[s], self.ge48[self.kind[s]], self.gs6[self.kind[s]]
            for dy, dx in itertools.product((-1, 0, 1), repeat=2):
                o = self.cxyz[s, :2] + torch.tensor([dx, dy], device=self.dev)
                wx, wy = o[:, 0] % nx, o[:, 1] % ny
                shift = torch.stack([o[:, 0] - wx, o[:, 1] - wy, torch.zeros_like(wx)], 1).double() * S.RS
                t = self.ctab[wx + nx * wy]
                d = p[:, None] - (self.carb[t] + shift[:, None])
                r2 = (d * d).sum(-1)
                i2 = 1.0 / r2
                i6 = i2 ** 3
                g = torch.where((t >= 0) & (r2 <= S.RC ** 2), e48[:, None] * i6 * (s6[:, None] * i6 - 0.5) * i2, 0.0)
                f[s] += (d * g[..., None]).sum(1)

    # velocity Verlet with the constraints met exactly
    def accel(self, f):
        self.a = f * (S.DT ** 2 / 2) / self.m[:, None]

    def _kinetic(self):
        return float((self.m[:, None] * self.v ** 2).sum()) / S.DT ** 2

    def _waters(self, t):
        return t[:3 * self.nw].view(-1, 3, 3)

    def _bonds(self, t):
        w = self._waters(t)
        return torch.stack([w[:, 0] - w[:, 1], w[:, 1] - w[:, 2], w[:, 2] - w[:, 0]], 1)

    def _push(self, t, g, r):
        """Adds the impulses g along the bond vectors r, over the masses, to the waters of t."""
        im = 1.0 / self.m[:3]
        d = g[..., None] * r
        self._waters(t).add_(torch.stack([d[:, 0] - d[:, 2], d[:, 1] - d[:, 0], d[:, 2] - d[:, 1]], 1) * im[:, None])

    def _matrix(self, p, r):
        im = 1.0 / self.m[:3]
        o, h = float(im[0]), float(im[1])
        k = torch.tensor([[o + h, -h, -o], [-h, 2 * h, -h], [-o, -h, o + h]], dtype=torch.float64, device=self.dev)
        return k * torch.einsum("nax,nbx->nab", p, r)

    def move_a(self):
        k1 = self._kinetic()
        es = 1.0 - self.eta * S.DT / 2
        old = self.x.clone()
        r = self._bonds(old)
        self.v = self.v * es + self.a
        self.x = self.x + self.v
        hh = 2.0 * math.sin(math.radians(109.47) / 2) / 3.166
        d2 = torch.tensor([1 / 3.166 ** 2, hh ** 2, 1 / 3.166 ** 2], dtype=torch.float64, device=self.dev)
        for _ in range(12):
            p = self._bonds(self.x)
            res = d2 - (p * p).sum(-1)
            g = torch.linalg.solve(2.0 * self._matrix(p, r), res[..., None])[..., 0]
            self._push(self.x, g, r)
            self._push(self.v, g, r)
        self.eta += self.pnh1 * (k1 + self.pnh2 + self._kinetic())

    def move_b(self, f):
        self.accel(f)
        self.v = 2.0 / (2.0 + self.eta * S.DT) * (self.v + self.a)
        r, u = self._bonds(self.x), self._bonds(self.v)
        g = torch.linalg.solve(self._matrix(r, r), -(r * u).sum(-1)[..., None])[..., 0]
        self._push(self.v, g, r)

    def temperature(self):
        return self._kinetic() / self.dof


def exact(case, seed):
    if case["preset"] != "config":
        return None
    out = []
    for s in _systems(case, seed):
        e = _Exact(s)
        if case["kind"] == "halves":
            acc, got = torch.tensor(_accelerations(case, [s], seed), device=e.dev), []
            for pos in (e.x, e.x + e.v):
                e.x, e.v, e.a, e.eta = pos, torch.tensor(s.vel, device=e.dev), acc, 0.0
                e.move_a()
                if not got:
                    e.rebuild()
                f = e.force()
                e.move_b(f)
                got += [f, e.x, e.v, e.a, torch.tensor([e.eta], dtype=torch.float64)]
            return [t.cpu() for t in got]
        e.rebuild()
        f = e.force()
        if case["kind"] == "force":
            e.x = e.x + e.v
            out.append([f, e.force()])
            continue
        e.accel(f)
        temps = []
        for kb in range(KB0, KB0 + STEPS):
            e.move_a()
            if kb % 10 == 0:
                e.rebuild()
            e.move_b(e.force())
            temps.append(e.temperature())
        out.append([e.x, e.v, e.a, torch.tensor(temps if case["kind"] == "loop" else [e.eta], dtype=torch.float64)])
    return [torch.cat([o[k].cpu() for o in out]) for k in range(len(out[0]))]
