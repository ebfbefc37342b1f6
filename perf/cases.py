"""Performance cases of the nonbonded engine: what a driver of this library has it do, through
the public entry points of ``mdcore_b200`` (the ctypes binding of the C API).

A case is one call pattern on one kind of system:

call      what one pass is
--------  ---------------------------------------------------------------------------------
force     ``Engine.nonbond``: one force evaluation, host particles in, host forces out
noalloc   ``engine_nonbond_cuda_noalloc``: one force evaluation on the caller's device buffers
step      ``Engine.step`` / ``Batch.step``: one ``engine_step``, host particles in and out
resident  ``resident_steps(steps)`` on the device, then the particles brought back to the host
minimize  the same with steepest-descent steps

system    particles (``size``)
--------  ---------------------------------------------------------------------------------
argon     LJ argon at liquid density, one table (``size``^3 FCC cells of 4 atoms)
water     rigid SPC/E water, three tables, exclusions, constraints (``size``^3 molecules)
slab      a two-type LJ liquid slab in its vapour, most cells nearly empty (``size`` atoms)
replicas  a batch of independent argon boxes of 500 to 8,000 atoms (``size`` boxes)
chains    solvated charged bead chains: 253 tables, per-particle charges, bonds, angles,
          dihedrals, rigid water (``size`` chains of 100 beads)

``tuned`` cases set the engine up as a long run does (CUDA graphs, the launch-shape
autotuner); the others run with the defaults, as a driver that only calls ``engine_step``.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "mdcore-history_b200"))
import mdcore_b200 as M  # noqa: E402
import workloads as W  # noqa: E402


# The stream of the calls on caller-owned device buffers: one for all of them, since they share
# one scratch area on the device and must not overlap.
_STREAM = torch.cuda.Stream() if torch.cuda.is_available() else None


def listed():
    return [
        # the smallest box the cell grid holds well, one force evaluation: latency of a call
        dict(name="argon-1372-force", call="force", system="argon", size=7),
        # a small solvent box stepped by a driver that keeps its particles on the host
        dict(name="water-3000-step", call="step", system="water", size=10),
        # forces for a host program that owns the device memory
        dict(name="argon-32000-noalloc", call="noalloc", system="argon", size=20),
        # a production run of a mid-sized simple liquid between two trajectory frames
        dict(name="argon-32000-resident", call="resident", system="argon", size=20, steps=100, tuned=True),
        # the same for an odd size with the default launch shape, no graphs
        dict(name="argon-8788-resident", call="resident", system="argon", size=13, steps=100, tuned=False),
        # rigid water at the size of a solvated protein: a production run (P-SHAKE), with frames
        # close together, since pairs that cross the cutoff decorrelate it fast
        dict(name="water-98304-resident", call="resident", system="water", size=32, steps=10, tuned=True),
        # the same through the drop-in engine_step, and with SHAKE at an odd size
        dict(name="water-98304-step", call="step", system="water", size=32),
        dict(name="water-36501-shake", call="resident", system="water", size=23, steps=10, tuned=True, shake=True),
        # heterogeneous solution: forces of a given configuration; relaxation of a new one
        dict(name="chains-40-force", call="force", system="chains", size=40),
        dict(name="chains-16-minimize", call="minimize", system="chains", size=16, steps=50, tuned=True),
        # a million atoms, inhomogeneous: most cells hold a few vapour atoms
        dict(name="slab-1048576-resident", call="resident", system="slab", size=1 << 20, steps=100, tuned=True),
        # an ensemble of replicas in one batch: the largest single-GPU job
        dict(name="replicas-512-resident", call="resident", system="replicas", size=512, steps=100, tuned=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["force", "noalloc", "step", "resident", "resident", "resident", "minimize"])
    if kind == "minimize":
        return dict(call=kind, system="chains", size=_log(rng, 12, 30), steps=rng.randint(20, 60),
                    tuned=rng.random() < 0.5)
    system = rng.choice({"force": ["argon", "water", "slab", "chains"], "noalloc": ["argon", "water"],
                         "step": ["argon", "water", "slab", "replicas"],
                         "resident": ["argon", "water", "slab", "replicas"]}[kind])
    big = kind == "resident"
    size = {"argon": lambda: _log(rng, 6, 30 if big else 20), "water": lambda: _log(rng, 10, 32 if kind != "noalloc" else 25),
            "slab": lambda: _log(rng, 20000, 700000 if big else 150000), "replicas": lambda: _log(rng, 3, 300 if big else 40),
            "chains": lambda: _log(rng, 12, 60)}[system]()
    case = dict(call=kind, system=system, size=size)
    if kind == "resident":
        case.update(steps=rng.randint(5, 10) if system == "water" else rng.randint(30, 100), tuned=rng.random() < 0.6)
        if system == "water":
            case["shake"] = rng.random() < 0.3
    return case


# ------------------------------------------------------------------------------- systems
def _hydrogen_bonded(s, seed):
    """The water with every molecule turned at random by some 15 degrees from the orientation in
    which its hydrogens face the oxygens of two neighbours (uniformly random orientations bring
    hydrogens into contact, and the first steps then throw molecules about)."""
    rng = np.random.default_rng(seed + 3)
    o = s.x[0::3]
    h = np.stack([s.x[1] - s.x[0], s.x[2] - s.x[0]])
    h -= np.round(h / s.dim) * s.dim
    angle = math.acos(float(h[0] @ h[1]) / 0.01)
    h = 0.1 * np.array([[1.0, 0.0, 0.0], [math.cos(angle), math.sin(angle), 0.0]])
    q = np.concatenate([np.ones((len(o), 1)), rng.normal(0.0, 0.08, size=(len(o), 3))], 1)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    w, u = q[:, None, :1], q[:, None, 1:]
    t = 2.0 * np.cross(u, h[None])
    turned = h[None] + w * t + np.cross(u, t)
    s.x = W.wrap_positions(np.concatenate([o[:, None], o[:, None] + turned], 1).reshape(-1, 3), s.dim)
    return s


def _systems(case, seed):
    """The case's systems (one, or the replicas): positions on jittered lattices, velocities of
    the temperature such a system is run at."""
    kind, size = case["system"], case["size"]
    if kind == "argon":
        s = [W.argon_fcc(size, seed=seed, jitter=0.02)]
        temperature = 100.0
    elif kind == "water":
        s = [W.with_rigid_water(_hydrogen_bonded(W.water_spce(size, seed=seed), seed), 300.0, seed=seed + 1)]
        temperature = None
    elif kind == "slab":
        # the full system's proportions: box 1 : 1 : 4, liquid on 7/40 of the height
        edge = 40.0 * (size / float(1 << 20)) ** (1.0 / 3.0)
        nx, nz = int(round(2.75 * edge)), int(round(77.0 / 40.0 * edge))
        s = [W.lj_slab(nx=nx, nz=nz, n_total=max(size, nx * nx * nz + 1), seed=seed, box=(edge, edge, 4 * edge),
                       slab=28.07 / 40.0 * edge)]
        temperature = 90.0
    elif kind == "replicas":
        # the ensemble's sizes and densities are the case's, the positions the seed's
        s = W.argon_replicas(size, seed=size)
        rng = np.random.default_rng(seed)
        for one in s:
            one.x = W.wrap_positions(one.x + rng.normal(0.0, 0.01, size=one.x.shape), one.dim)
        temperature = 100.0
    else:
        # a fixed volume per chain with its share of water; to be relaxed, a calmer contact
        # distance, which fewer waters keep, and no angles or dihedrals
        edge = max(3.65, (4.135 * size) ** (1.0 / 3.0))
        relax = case["call"] == "minimize"
        s = [W.chains_water(nchains=size, length=100, nwater=(50 if relax else 70) * size, box=(edge, edge, edge),
                            seed=seed, gap=0.25 if relax else 0.2, angles_dihedrals=not relax)]
        temperature = None
    if case["call"] in ("step", "resident") and temperature is not None:
        for k, one in enumerate(s):
            one.v = W.maxwell_velocities(one, temperature, seed=seed + 7 + k)
    return s


def _bin(s):
    """Cell of every particle and its position relative to the cell, the engine's storage."""
    cdim = np.floor(s.dim / s.L).astype(np.int64)
    h = s.dim / cdim
    ind = ((s.x - s.origin) * (1.0 / h)).astype(np.int64)
    return cdim, h, ind, (s.x - (s.origin + ind * h)).astype(np.float32)


def _slots(n, ncells):
    """Room for n particles in cells padded to multiples of four, whatever they hold."""
    return (n + 3 * ncells + 3) // 4 * 4


def prepare(case, seed):
    systems = _systems(case, seed)
    state = dict(case=case, n=[s.n for s in systems])
    flags = M.engine_flag_cuda | (M.engine_flag_shake if case.get("shake") else 0)
    if case["system"] == "replicas":
        state["engines"] = [M.Engine.from_system(s, flags=flags, start=False) for s in systems]
        state["e"] = M.Batch(state["engines"], device=0)
    else:
        state["e"] = M.Engine.from_system(systems[0], flags=flags)
        state["engines"] = [state["e"]]
    e = state["e"]
    if case.get("tuned"):
        e.graph(True)
        e.load_parts()
        e.autotune(5)
    if case["call"] == "minimize":
        e.minimize(2e-7, 0.002)
    if case["call"] in ("resident", "minimize"):
        e.resident_begin()
    if case["call"] == "noalloc":
        s = systems[0]
        cdim, _, ind, xrel = _bin(s)
        cell = (ind[:, 0] * cdim[1] + ind[:, 1]) * cdim[2] + ind[:, 2]
        ncells = int(np.prod(cdim))
        count = np.bincount(cell, minlength=ncells).astype(np.int32)
        start = np.zeros(ncells + 1, np.int32)
        start[1:] = np.cumsum((count + 3) // 4 * 4)
        nslots = _slots(s.n, ncells)
        order = np.argsort(cell, kind="stable")
        first = np.concatenate([[0], np.cumsum(count)])[:-1]
        slot = start[cell[order]] + (np.arange(s.n) - first[cell[order]])
        xq = np.zeros((nslots, 4), np.float32)
        pid = np.zeros(nslots, np.int32)
        xq[slot, :3] = xrel[order]
        xq.view(np.int32)[slot, 3] = s.type[order]
        pid[slot] = order
        dev = torch.device("cuda", 0)
        state["buf"] = [torch.from_numpy(a).to(dev) for a in (xq, pid, start, count)]
        state["maxcount"] = int(count.max())
        state["force"] = torch.zeros(3 * len(pid), dtype=torch.int64, device=dev)
        state["epot"] = torch.zeros(ncells, dtype=torch.int64, device=dev)
        state["acc"] = torch.zeros(8, dtype=torch.int64, device=dev)
        torch.cuda.current_stream().synchronize()     # the buffers are used on another stream
        fn = M.lib().engine_nonbond_cuda_noalloc
        fn.restype = ctypes.c_int
        fn.argtypes = [ctypes.c_void_p] * 5 + [ctypes.c_int] * 2 + [ctypes.c_void_p] * 4
        state["fn"] = fn
    if case["call"] in ("resident", "minimize"):
        # what a trajectory writer keeps: the particle buffers it reads into, and where the
        # displacements are counted from
        n = sum(state["n"])
        state["x"], state["v"], state["f"], state["moved"] = (np.zeros((n, 3), np.float32) for _ in range(4))
        state["cell"] = np.zeros(n, np.int32)
        grids = [_bin(s) for s in systems]
        state["grid"] = [(g[0], g[1], s.dim) for g, s in zip(grids, systems)]
        state["cell0"] = np.concatenate([(g[2][:, 0] * g[0][1] + g[2][:, 1]) * g[0][2] + g[2][:, 2] for g in grids])
        state["cell0"] = state["cell0"].astype(np.int32)
        state["x0"] = np.concatenate([g[3] for g in grids])
    return state


# ------------------------------------------------------------------------------- one pass
def _read(state):
    """Every particle by id: displacement from the start (the nearest image, as for a mean-square
    displacement, so that neither cells nor the box's faces show), velocity, force."""
    at = 0
    for e, n in zip(state["engines"], state["n"]):
        M._check(e.lib.engine_getparts(e.ptr, state["x"][at:].ctypes.data, state["v"][at:].ctypes.data,
                                       state["f"][at:].ctypes.data, state["cell"][at:].ctypes.data, n), "engine_getparts")
        at += n
    moved = np.subtract(state["x"], state["x0"], out=state["moved"])
    left = np.flatnonzero(state["cell"] != state["cell0"])
    at = 0
    for (cdim, h, dim), n in zip(state["grid"], state["n"]):
        k = left[np.searchsorted(left, at):np.searchsorted(left, at + n)]
        now, was = state["cell"][k], state["cell0"][k]
        d = np.stack([now // (cdim[1] * cdim[2]) - was // (cdim[1] * cdim[2]),
                      now // cdim[2] % cdim[1] - was // cdim[2] % cdim[1], now % cdim[2] - was % cdim[2]], 1) * h
        d += moved[k]
        moved[k] = d - np.round(d / dim) * dim
        at += n
    return dict(moved=moved, v=state["v"], f=state["f"])


def run(state):
    case, e = state["case"], state["e"]
    if case["call"] == "force":
        e.nonbond()
        st = e.stats()
        return dict(f=e.forces(), epot=st.epot, virial=st.virial, pairs=int(st.pairs), excluded=int(st.excluded),
                    candidates=int(st.candidates))
    if case["call"] == "noalloc":
        xq, pid, start, count = state["buf"]
        with torch.cuda.stream(_STREAM):
            M._check(state["fn"](e.ptr, xq.data_ptr(), pid.data_ptr(), start.data_ptr(), count.data_ptr(), len(pid),
                                 state["maxcount"], state["force"].data_ptr(), state["epot"].data_ptr(),
                                 state["acc"].data_ptr(), _STREAM.cuda_stream), "engine_nonbond_cuda_noalloc")
            return dict(f=state["force"] * 2.0 ** -24, epot=state["epot"] * 2.0 ** -32, count=state["acc"][2:6].clone())
    if case["call"] == "step":
        e.step()
        return [np.concatenate(a) for a in zip(*[one.parts() for one in state["engines"]])]
    e.resident_steps(case["steps"])
    e.resident_sync()
    return _read(state)


# ------------------------------------------------------------------------------- limits
def _density(case):
    """(particles, particles per nm^3 where the pairs are, cutoff) of the case."""
    k, size = case["system"], case["size"]
    if k == "argon":
        return 4 * size ** 3, 21.0, 1.0
    if k == "water":
        return 3 * size ** 3, 100.2, 1.0
    if k == "slab":
        return size, 17.2, 1.0          # averaged over the particles (liquid 21, vapour 0.55)
    if k == "replicas":
        return 2835 * size, 19.4, 1.0   # 500 to 8,000 atoms each, 18 to 24 per nm^3
    if case["call"] == "minimize":
        return 250 * size, 60.0, 1.2
    return 310 * size, 75.0, 1.2


def work(case):
    """45 FP32 operations per pair within the cutoff (displacement, distance, table, forces),
    each particle's state read and written once per pass."""
    n, rho, rc = _density(case)
    steps = case.get("steps", 1)
    pairs = n * rho * 2.0 / 3.0 * math.pi * rc ** 3
    return dict(bytes=float(n * (20 + 24 if case["call"] in ("force", "noalloc") else 32 + 40)), flops=45.0 * pairs * steps)


def tolerance(case):
    """About four times what the same evaluation in another order of its sums (the other lane
    layout) shows after two passes; one evaluation: what FP32 pair arithmetic shows against 64
    bits.  In water and chains a pair that crosses the cutoff one step earlier or later gives
    its particles a kick (truncated Coulomb forces), which a trajectory then carries on."""
    if case["call"] in ("force", "noalloc"):
        return dict(rel=1e-5, max=2e-4)
    if case["call"] == "step":
        return dict(rel=6e-4, max=0.15)
    if case["call"] == "minimize":
        return dict(rel=5e-4, max=0.02)
    if case["system"] == "water":
        return dict(rel=1e-2, max=0.9)
    return dict(rel=2e-4, max=0.03)


# ------------------------------------------------------------------------------- 64 bits
def _tables(s):
    """The case's potential tables, an input of the path: per table its interval polynomial and
    coefficients in 64 bits, and the table of every type pair."""
    dev = torch.device("cuda", 0)
    mt = len(s.masses)
    idx = torch.full((mt, mt), -1, dtype=torch.int64, device=dev)
    alpha, coef, base, last = [], [], [], []
    at = 0
    for k, spec in enumerate(list(s.pots) + ([s.ep] if s.ep is not None else [])):
        n, a, c = M.create_potential(spec).contents.table()
        if k < len(s.pots):
            idx[spec.ti, spec.tj] = idx[spec.tj, spec.ti] = k
        alpha.append(a[:3])
        coef.append(c.reshape(-1, 8))
        base.append(at)
        last.append(n)
        at += n + 1
    f64 = dict(dtype=torch.float64, device=dev)
    return dict(idx=idx, alpha=torch.tensor(np.array(alpha), **f64), coef=torch.tensor(np.concatenate(coef), **f64),
                base=torch.tensor(base, device=dev), last=torch.tensor(last, device=dev))


def _look_up(t, k, r):
    a = t["alpha"][k]
    i = (a[:, 0] + r * (a[:, 1] + r * a[:, 2])).clamp(min=0.0).to(torch.int64)
    c = t["coef"][t["base"][k] + torch.minimum(i, t["last"][k])]
    x = (r - c[:, 0]) * c[:, 1]
    e, d = c[:, 2] * x + c[:, 3], c[:, 2]
    for q in range(4, 8):
        d = d * x + e
        e = e * x + c[:, q]
    return e, d * c[:, 1] / r


def _near(x, dim, reach, rows=512):
    """Index pairs i < j within `reach` (nearest images)."""
    n = len(x)
    out = []
    rows = max(1, min(n, (rows * 65536) // max(1, n)))
    for a in range(0, n, rows):
        d = x[a:a + rows, None, :].float() - x[None, a:, :].float()
        d -= torch.round(d / dim.float()) * dim.float()
        i, j = torch.nonzero((d * d).sum(-1) < reach * reach, as_tuple=True)
        keep = j > i
        out.append(torch.stack([i[keep] + a, j[keep] + a]))
    return torch.cat(out, 1)


class _Exact:
    """Nonbonded forces of one system in 64 bits."""

    def __init__(self, s):
        dev = torch.device("cuda", 0)
        _, h, ind, xrel = _bin(s)
        self.x = torch.from_numpy(s.origin + ind * h + xrel.astype(np.float64)).to(dev)
        self.dim = torch.from_numpy(np.asarray(s.dim, np.float64)).to(dev)
        self.type = torch.from_numpy(np.asarray(s.type, np.int64)).to(dev)
        self.q = None if s.ep is None else torch.from_numpy(np.asarray(s.q, np.float32).astype(np.float64)).to(dev)
        self.cut = s.cutoff
        self.tab = _tables(s)
        self.n = s.n
        ex = np.sort(np.asarray(s.excl, np.int64).reshape(-1, 2), 1)
        self.excl = torch.from_numpy(ex[:, 0] * s.n + ex[:, 1]).to(dev)
        self.list_x = None

    def pairs(self):
        skin = 0.12
        moved = None if self.list_x is None else (self.x - self.list_x).square().sum(-1).max().sqrt().item()
        if moved is None or 2.0 * moved > skin:
            ij = _near(self.x, self.dim, self.cut + skin + 1e-3)
            if len(self.excl):
                ij = ij[:, ~torch.isin(ij[0] * self.n + ij[1], self.excl)]
            self.list, self.list_x = ij, self.x.clone()
        return self.list

    def forces(self):
        ij = self.pairs()
        f = torch.zeros_like(self.x)
        epot = virial = 0.0
        for a in range(0, ij.shape[1], 1 << 23):
            i, j = ij[0, a:a + (1 << 23)], ij[1, a:a + (1 << 23)]
            d = self.x[i] - self.x[j]
            d -= torch.round(d / self.dim) * self.dim
            r2 = (d * d).sum(-1)
            k = self.tab["idx"][self.type[i], self.type[j]]
            on = (r2 <= self.cut * self.cut) & ((k >= 0) | (self.q is not None))
            i, j, d, k, r = i[on], j[on], d[on], k[on], r2[on].sqrt()
            e, g = _look_up(self.tab, k.clamp(min=0), r)
            e, g = torch.where(k >= 0, e, 0.0), torch.where(k >= 0, g, 0.0)
            if self.q is not None:
                qq = self.q[i] * self.q[j]
                ee, ge = _look_up(self.tab, torch.full_like(k, len(self.tab["base"]) - 1), r)
                e, g = e + qq * ee, g + qq * ge
            w = g[:, None] * d
            f.index_add_(0, i, -w)
            f.index_add_(0, j, w)
            epot += e.sum().item()
            virial -= (w * d).sum().item()
        return f, epot, virial


def exact(case, seed):
    n = _density(case)[0]
    if case["system"] == "slab" and n > 100000 or n > 120000 and case["system"] != "replicas":
        return None
    if case["call"] in ("force", "noalloc"):
        s = _systems(case, seed)[0]
        f, epot, virial = _Exact(s).forces()
        if case["call"] == "force":
            return dict(f=f.cpu().numpy(), epot=epot, virial=virial, pairs=None, excluded=None, candidates=None)
        cdim, _, ind, _ = _bin(s)
        cell = (ind[:, 0] * cdim[1] + ind[:, 1]) * cdim[2] + ind[:, 2]
        count = np.bincount(cell, minlength=int(np.prod(cdim)))
        start = np.concatenate([[0], np.cumsum((count + 3) // 4 * 4)])
        order = np.argsort(cell, kind="stable")
        first = np.concatenate([[0], np.cumsum(count)])[:-1]
        out = np.zeros((_slots(s.n, len(count)), 3))
        out[start[cell[order]] + (np.arange(s.n) - first[cell[order]])] = f.cpu().numpy()[order]
        return dict(f=out.reshape(-1), epot=None, count=None)
    # trajectories: the systems without constraints, of a size that lists of pairs serve
    if case["call"] != "resident" or case["system"] not in ("argon", "replicas") or n * case["steps"] > 2e7:
        return None
    moved, vel, force = [], [], []
    for s in _systems(case, seed):
        x = _Exact(s)
        v = torch.from_numpy(np.asarray(s.v, np.float64).astype(np.float32).astype(np.float64)).to(x.x.device)
        dt = float(np.float32(s.dt))
        w = torch.from_numpy(np.float32(dt / np.asarray(s.masses)).astype(np.float64)).to(x.x.device)[x.type][:, None]
        x0 = torch.from_numpy(s.x).to(x.x.device)
        for _ in range(case["steps"]):
            f = x.forces()[0]
            v = v + f * w
            x.x = x.x + dt * v
        d = x.x - x0
        moved.append((d - torch.round(d / x.dim) * x.dim).cpu())
        vel.append(v.cpu())
        force.append(f.cpu())
    return dict(moved=torch.cat(moved), v=torch.cat(vel), f=torch.cat(force))
