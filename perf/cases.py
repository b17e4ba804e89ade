"""The work that programs have this package do, as cases that can be timed.

Each case is one call pattern of a user of the fix: an engine that drives the
hooks with its own host arrays, a driver that runs device-resident steps from
a given state, batched replicas, full MD with the eam/alloy pair force, a
fitting loop's forward and backward pass, and the grid solve on a caller's own
device arrays.  `prepare` makes the inputs from a seed and the context such a
program keeps; `run` is one pass; `exact` restates the same pass in FP64
torch without the package.

Inputs are fcc Ni lattices at a temperature with Gaussian jitter, the synthetic
beta file of the package's workloads (or the quadratic one its fitting uses)
and the Ni.eam setfl file kept with the tests; sizes run from a few hundred
atoms (a unit test's box) to the benchmark's two million.
"""
from __future__ import annotations

import ctypes
import lzma
import math
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "user-eph_gb300"))

import ephgb  # noqa: E402
from ephgb import workloads as W  # noqa: E402
from ephgb.adjoint import Adjoint  # noqa: E402

DEVICE = "cuda"
NI_EAM = os.path.join(ROOT, "tests", "golden", "ref_inputs", "MD_Run_Ni.eam.xz")
A0 = W.NI_LATTICE
RHO_E, C_E, KAPPA = 1.0, 3.5e-6, 0.1
FE_MASS = 55.845


def _steps(cells, grid, steps, **more):
    case = dict(kind="steps", nx=cells[0], ny=cells[1], nz=cells[2], gx=grid[0], gy=grid[1], gz=grid[2], steps=steps,
                mode="fast", pairs="df64", elements=1, outside=0.0, T_e=300.0, pka=0.0, dt=0.001, graph=False)
    case.update(more)
    return case


def listed():
    def named(name, case):
        return dict(case, name=name)

    return [
        # an engine stepping a unit-test box through the hooks, its own
        # Gaussian stream handed in: launches, copies and waits are the cost
        named("hooks_500", dict(kind="hooks", nx=5, ny=5, nz=5, gx=5, gy=5, gz=5, T_e=300.0, dt=0.001, xi="host")),
        # an engine's step at a production size: x and f in, f and the
        # per-atom array out, device deviates
        named("hooks_500k", dict(kind="hooks", nx=50, ny=50, nz=50, gx=40, gy=40, gz=40, T_e=300.0, dt=0.0005,
                                 xi="device")),
        # the CPU-runnable configuration (10^3 cells, 10^3 grid), from a state
        named("steps_4k", _steps((10, 10, 10), (10, 10, 10), 10)),
        # an uneven alloy box with part of the atoms outside the fix group,
        # steps replayed from a graph
        named("steps_ragged_alloy", _steps((13, 11, 17), (9, 7, 13), 10, elements=2, outside=0.2, T_e=900.0, graph=True)),
        # the equilibration runs: hot electrons, ions at 300 K
        named("steps_32k", _steps((20, 20, 20), (16, 16, 16), 10, T_e=2000.0)),
        # an alloy cascade of middle size
        named("steps_131k_alloy", _steps((32, 32, 32), (26, 26, 26), 10, elements=2, pka=5000.0, dt=0.0005)),
        # the bit-for-bit arithmetic, for those who check against the reference
        named("exact_62k", _steps((25, 25, 25), (20, 20, 20), 4, mode="exact")),
        # the benchmark's cascade
        named("cascade_2m", _steps((80, 80, 80), (64, 64, 64), 10, pka=10000.0, dt=0.0005)),
        # independent cascades stepped together
        named("batch_16", dict(kind="batch", replicas=16, least=20, most=30, steps=5, dt=0.0005)),
        # full MD: eam/alloy pair force and the fix
        named("md_256k", dict(kind="md", nx=40, ny=40, nz=40, gx=32, gy=32, gz=32, steps=5, T_e=300.0, pka=5000.0,
                              dt=0.0005)),
        # one iteration of a fit: forward, backward, the knot gradients
        named("gradient_32k", dict(kind="gradient", nx=20, ny=20, nz=20, gx=16, gy=16, gz=16, steps=20, every=10,
                                   T_e=2000.0, dt=0.001)),
        # the grid solve alone on a caller's arrays, with walls and sources
        named("grid_64", dict(kind="grid", gx=64, gy=64, gz=64, box=225.28, dt=0.002, walls=True)),
    ]


def draw(rng):
    def size(lo, hi):
        """about the same number on every axis, log-uniform, a cell or two apart"""
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return [max(lo, min(hi, int(round(n * rng.uniform(0.85, 1.18))))) for _ in range(3)]

    kind = rng.choice(["steps", "steps", "steps", "steps", "hooks", "hooks", "batch", "md", "gradient", "grid"])
    dt = rng.choice([0.0005, 0.001])
    T_e = round(math.exp(rng.uniform(math.log(250.0), math.log(5000.0))), 1)
    if kind == "steps":
        mode = rng.choice(["fast", "fast", "fast", "exact"])
        c = size(5, 72 if mode == "fast" else 32)
        g = [max(2, min(64, int(round(0.8 * k * rng.uniform(0.8, 1.25))))) for k in c]
        return _steps(c, g, rng.choice([4, 7, 10]), mode=mode, pairs=rng.choice(["df64", "df64", "df64", "fp64"]),
                      elements=rng.choice([1, 1, 2]), outside=rng.choice([0.0, 0.0, 0.3]), T_e=T_e,
                      pka=rng.choice([0.0, 2000.0, 10000.0]), dt=dt, graph=rng.random() < 0.5)
    if kind == "batch":
        least = rng.randint(8, 24)
        return dict(kind=kind, replicas=rng.randint(3, 24), least=least, most=least + rng.randint(2, 8), steps=rng.randint(3, 8),
                    dt=dt)
    if kind == "gradient":
        c = size(8, 24)
        every = rng.randint(4, 12)
        return dict(kind=kind, nx=c[0], ny=c[1], nz=c[2], gx=rng.randint(6, 16), gy=rng.randint(6, 16),
                    gz=rng.randint(6, 16), steps=every * 2 + rng.randint(0, 3), every=every, T_e=T_e, dt=dt)
    if kind == "grid":
        g = size(8, 64)
        return dict(kind=kind, gx=g[0], gy=g[1], gz=g[2], box=round(3.52 * sum(g) / 3.0, 2), dt=rng.choice([0.001, 0.002]),
                    walls=rng.random() < 0.5)
    if kind == "hooks":
        c = size(5, 50)
        return dict(kind=kind, nx=c[0], ny=c[1], nz=c[2], gx=max(2, c[0] * 4 // 5), gy=max(2, c[1] * 4 // 5),
                    gz=max(2, c[2] * 4 // 5), T_e=T_e, dt=dt, xi=rng.choice(["host", "device"]))
    c = size(8, 48)
    return dict(kind="md", nx=c[0], ny=c[1], nz=c[2], gx=max(2, c[0] * 4 // 5), gy=max(2, c[1] * 4 // 5),
                gz=max(2, c[2] * 4 // 5), steps=rng.randint(3, 6), T_e=T_e, pka=rng.choice([0.0, 5000.0]), dt=0.0005)


# ------------------------------------------------------------------ inputs


def _beta_file(case, folder):
    path = os.path.join(folder, "synth.beta")
    if case["kind"] == "gradient":  # the fitting workload's file: few knots, beta with curvature
        return W.write_beta_file(path, n_rho=16, n_beta=64, drho=0.02, beta_fn=lambda r: 0.02 + 2.0 * r * r)
    if case.get("elements", 1) == 2:
        return W.write_beta_file(path, elements=("Ni", "Fe"), numbers=(28, 26))
    return W.write_beta_file(path)


def _system(case, seed, folder):
    """The fix words and atoms of a case."""
    atoms = W.fcc_lattice((case["nx"], case["ny"], case["nz"]), seed=seed)
    rng = np.random.default_rng([seed, 1])
    elements = ("Ni",)
    if case.get("elements", 1) == 2:
        elements = ("Ni", "Fe")
        atoms.type = np.where(rng.random(atoms.n) < 0.3, 2, 1).astype(np.int32)
        atoms.mass = np.array([0.0, W.NI_MASS, FE_MASS])
    if case.get("outside", 0.0) > 0.0:
        atoms.mask = np.where(rng.random(atoms.n) < case["outside"], 2, 1).astype(np.int32)
    if case.get("pka", 0.0) > 0.0:
        W.add_pka(atoms, case["pka"], seed=seed + 1)
    words = W.fix_args(_beta_file(case, folder), seed=1 + seed % 900000, flags=15 if case["kind"] == "hooks" else 7,
                       rho_e=RHO_E, C_e=C_E, kappa_e=KAPPA, T_e=case["T_e"], grid=(case["gx"], case["gy"], case["gz"]),
                       T_out=os.path.join(folder, "Te_out"), elements=elements)
    return words, atoms


def _grid_T(case, seed):
    """An electronic temperature field around T_e."""
    n = case["gx"] * case["gy"] * case["gz"]
    return case["T_e"] * np.random.default_rng([seed, 2]).uniform(0.9, 1.1, n)


def _start_force(n, seed):
    return np.random.default_rng([seed, 3]).normal(0.0, 0.05, (n, 3))


def _grid_arrays(case, seed):
    """A caller's grid: temperatures, a source, parameters that vary by cell;
    with walls a ZERO_DERIVATIVE plane and a CONSTANT line."""
    rng = np.random.default_rng([seed, 4])
    n = (case["gx"], case["gy"], case["gz"])
    k, j, i = np.meshgrid(np.arange(n[2]), np.arange(n[1]), np.arange(n[0]), indexing="ij")
    flag = np.ones(i.size, dtype=np.int8)
    if case["walls"]:
        flag[(i == 0).ravel()] = 2
        flag[((j == 0) & (k == 0) & (i > 0)).ravel()] = 0
    t = i.size
    return dict(T=rng.uniform(200.0, 2000.0, t), dT=rng.uniform(-0.5, 0.5, t), S=rng.uniform(0.0, 0.1, t),
                rho=rng.uniform(0.9, 1.1, t), C=rng.uniform(3e-6, 4e-6, t), kappa=rng.uniform(0.05, 0.1, t), flag=flag)


class State:
    """What a program keeps between passes."""


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE)


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory()


def _restart_of(s, atoms, T, f):
    s.x, s.v, s.f, s.T = _device(atoms.x), _device(atoms.v), _device(f), _device(T)
    s.out = {k: torch.empty_like(getattr(s, k)) for k in ("x", "v", "f", "T")}


def _put_state(fix, s):
    for k in ("x", "v", "f", "T"):
        fix.put(k, getattr(s, k))


def _get_state(fix, s):
    for k in ("x", "v", "f", "T"):
        fix.get(k, s.out[k])
    return dict(s.out)


def prepare(case, seed):
    s = State()
    s.case, kind = case, case["kind"]
    s.folder = tempfile.TemporaryDirectory()
    if kind == "grid":
        a = _grid_arrays(case, seed)
        s.host = dict(lo=np.zeros(3), hi=np.array([case["box"]] * 3))
        s.dev = {k: _device(v) for k, v in a.items()}
        s.T0 = s.dev["T"].clone()
        s.nsub = ctypes.c_uint()
        return s
    if kind == "batch":
        s.parts = []
        replicas = []
        for r, c in enumerate(_replica_cases(case)):
            words, atoms = _system(c, seed + 101 * r, s.folder.name)
            part = State()
            _restart_of(part, atoms, _grid_T(c, seed + 101 * r), _start_force(atoms.n, seed + 101 * r))
            s.parts.append(part)
            replicas.append((words, atoms))
        s.batch = ephgb.Batch(replicas, dt=case["dt"])
        return s
    words, atoms = _system(case, seed, s.folder.name)
    eam = None
    if kind == "md":
        path = os.path.join(s.folder.name, "Ni.eam")
        with open(NI_EAM, "rb") as src, open(path, "wb") as dst:
            dst.write(lzma.decompress(src.read()))
        eam = (path, ["Ni"])
    mode = ephgb.MODE_EXACT if case.get("mode") == "exact" else ephgb.MODE_FAST
    s.fix = ephgb.FixEPH(words, atoms, dt=case["dt"], mode=mode, eam=eam)
    if case.get("pairs") == "fp64":
        s.fix.set_pair_arithmetic(ephgb.PAIRS_FP64)
    if case.get("graph"):
        s.fix.set_graph(True)
    if kind == "gradient":
        s.adjoint = Adjoint(s.fix, checkpoint_every=case["every"])
        s.knots = s.adjoint.columns[0][1] * (1.0 + 0.1 * np.sin(np.arange(64) / (4.0 + seed % 5)))
        s.dE, s.dT = _cotangents(case, seed)
    elif kind == "hooks":
        s.x, s.v, s.f0 = _pinned(atoms.x), _pinned(atoms.v), _pinned(_start_force(atoms.n, seed))
        s.f, s.array = _pinned(np.zeros((atoms.n, 3))), _pinned(np.zeros((atoms.n, 8)))
        s.xi = _pinned(_host_xi(atoms.n, seed)) if case["xi"] == "host" else None
        s.T, s.T_out = _device(_grid_T(case, seed)), _device(_grid_T(case, seed))
    else:
        _restart_of(s, atoms, _grid_T(case, seed), _start_force(atoms.n, seed))
    return s


def _replica_cases(case):
    """Replica r of a batch: cells and grid spread over the batch's range."""
    for r in range(case["replicas"]):
        n = case["least"] + (r * (case["most"] - case["least"])) // max(1, case["replicas"] - 1)
        g = max(4, int(round(16 + (n - 20) * 32.0 / 30.0)))
        yield dict(kind="steps", nx=n, ny=n, nz=n, gx=g, gy=g, gz=g, T_e=300.0, pka=1000.0 + 500.0 * r, dt=case["dt"],
                   steps=case["steps"])


def _host_xi(n, seed):
    return np.random.default_rng([seed, 5]).standard_normal((n, 3))


def _cotangents(case, seed):
    rng = np.random.default_rng([seed, 6])
    return rng.uniform(-1.0, 1.0, case["steps"]), rng.uniform(-1.0, 1.0, case["steps"]) * 1e-2


# -------------------------------------------------------------------- passes


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "grid":
        d = s.dev
        d["T"].copy_(s.T0)
        p = {k: ctypes.c_void_p(t.data_ptr()) for k, t in d.items()}
        rc = ephgb.lib().eph_fdm_solve_noalloc(
            case["gx"], case["gy"], case["gz"], s.host["lo"].ctypes.data_as(ephgb._dp),
            s.host["hi"].ctypes.data_as(ephgb._dp), case["dt"], 1, p["T"], p["dT"], p["S"], p["rho"], p["C"],
            p["kappa"], p["flag"], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.byref(s.nsub))
        if rc:
            raise ephgb.EphError(rc, "grid solve")
        return {"T": d["T"], "substeps": s.nsub.value}
    if kind == "batch":
        for rep, part in zip(s.batch.replicas, s.parts):
            _put_state(rep, part)
        for rep in s.batch.replicas:
            rep.synchronize()  # the batch steps on a stream of its own
        s.batch.step(case["steps"])
        s.batch.synchronize()
        return [{k: v for k, v in _get_state(rep, part).items() if k in ("x", "v")}
                for rep, part in zip(s.batch.replicas, s.parts)]
    if kind == "gradient":
        s.adjoint.set_knots(0, beta_knots=s.knots)
        E, T = s.adjoint.forward(case["steps"])
        s.adjoint.backward(s.dE, s.dT)
        return dict(s.adjoint.gradients(0), E=E, T=T)
    if kind == "hooks":
        s.fix.put("T", s.T)
        s.fix.post_force_host(s.x.numpy(), s.f.numpy(), s.array.numpy(), xi=None if s.xi is None else s.xi.numpy(),
                              f_in=s.f0.numpy())
        s.fix.put("v", s.v.numpy())
        s.fix.end_of_step()
        return {"f": s.f, "array": s.array, "T": s.fix.get("T", s.T_out)}
    _put_state(s.fix, s)
    s.fix.step(case["steps"])
    out = _get_state(s.fix, s)
    if kind == "md":
        out["pair_energy"] = s.fix.pair_energy()
    return out


def work(case):
    """Per pass: every atom's x, v, f read and written once a step, the grid
    once; ~80 operations per pair and step for the fix, ~120 with the pair
    force (twice as many pairs), ~30 per cell and substep."""
    kind = case["kind"]
    if kind == "grid":
        cells = case["gx"] * case["gy"] * case["gz"]
        return {"bytes": 57.0 * cells, "flops": 30.0 * cells * _grid_substeps(case)}
    if kind == "batch":
        parts = [work(c) for c in _replica_cases(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, cells = 4 * case["nx"] * case["ny"] * case["nz"], case["gx"] * case["gy"] * case["gz"]
    per_pair = 80.0 * 42.0 + (120.0 * 78.0 if kind == "md" else 0.0)
    steps = case.get("steps", 1) * (3 if kind == "gradient" else 1)
    return {"bytes": steps * (144.0 * n + 16.0 * cells), "flops": steps * (n * (per_pair + 200.0) + 150.0 * cells)}


def _grid_substeps(case):
    h2 = sum((g / case["box"]) ** 2 for g in (case["gx"], case["gy"], case["gz"]))
    return max(1, int(case["dt"] * h2 * 0.1 / (0.4 * 3e-6 * 0.9)))


# ------------------------------------------- the same passes in FP64 torch


def _spline(dx, y):
    """Coefficients (a, b, c, d per interval, in powers of x) of the fix's
    spline through knots y (a tensor: differentiable in y)."""
    n = y.numel()
    b = (y[1:] - y[:-1]) / dx
    z1 = 2.0 * b[0] - b[1]
    z0 = 2.0 * z1 - b[0]
    z2 = 2.0 * b[n - 2]
    b = torch.cat([b, z2.reshape(1)])  # slope of each interval, and past the last
    after = torch.cat([b[1:], torch.zeros_like(z2).reshape(1)])
    before = torch.cat([z1.reshape(1), b[:-1]])
    before2 = torch.cat([z0.reshape(1), z1.reshape(1), b[:-2]])
    w1 = torch.cat([(b[1:] - b[:-1]).abs(), z2.abs().reshape(1)])  # the slope after that is 2 z2
    w0 = (before - before2).abs()
    total = w0 + w1
    ok = total > 0
    s = torch.where(ok, (before * w1 + b * w0) / torch.where(ok, total, torch.ones_like(total)), b)
    s = torch.where((before2 == before) & (b != after), before, s)
    s = torch.where((before == b) & (before2 != before), b, s)
    i = torch.arange(n - 1, dtype=y.dtype)
    x0, x1 = i * dx, (i + 1) * dx
    p0, p1 = x0 * x0, x1 * x1
    q0, q1 = x0 * p0, x1 * p1
    a0, a1, y0, y1 = s[:-1], s[1:], y[:-1], y[1:]
    d = (-a0 * x0 - a1 * x0 + a0 * x1 + a1 * x1 + 2.0 * y0 - 2.0 * y1) / (dx * dx * dx)
    c = (-a0 + a1 + 3.0 * d * p0 - 3.0 * d * p1) / 2.0 / dx
    bb = (c * p0 + d * q0 - c * p1 - d * q1 - y0 + y1) / dx
    a = y0 - bb * x0 - c * p0 - d * q0
    last = torch.stack([y[-1], torch.zeros_like(y[-1]), torch.zeros_like(y[-1]), torch.zeros_like(y[-1])])
    return torch.cat([torch.stack([a, bb, c, d], 1), last.reshape(1, 4)])


def _eval(table, dx, x):
    c = table[(x * (1.0 / dx)).long().clamp(0, table.shape[0] - 1)]
    return c[..., 0] + x * (c[..., 1] + x * (c[..., 2] + x * c[..., 3]))


class _Tables:
    """rho(r^2), beta(rho) and alpha(rho) of a beta file's columns."""

    def __init__(self, path):
        with open(path) as f:
            lines = f.read().split("\n")
        names = lines[3].split()[1:]
        tok = " ".join(lines[4:]).split()
        self.n_rho, self.dr, self.n_beta, self.drho, self.rc = int(tok[0]), float(tok[1]), int(tok[2]), float(tok[3]), float(tok[4])
        self.columns, at = [], 5
        for _ in names:
            r = torch.tensor([float(v) for v in tok[at + 1:at + 1 + self.n_rho]], dtype=torch.float64)
            b = torch.tensor([float(v) for v in tok[at + 1 + self.n_rho:at + 1 + self.n_rho + self.n_beta]],
                             dtype=torch.float64)
            self.columns.append((r, b))
            at += 1 + self.n_rho + self.n_beta
        self.build()

    def build(self):
        self.dr2 = self.rc ** 2 / (self.n_rho - 1)
        self.rho_max = self.drho * (self.n_beta - 1)
        r = torch.sqrt(torch.arange(self.n_rho, dtype=torch.float64) * self.dr2)
        self.rho = [_spline(self.dr2, _eval(_spline(self.dr, k), self.dr, r)).to(DEVICE) for k, _ in self.columns]
        self.alpha = [_spline(self.drho, torch.sqrt(k)).to(DEVICE) for _, k in self.columns]
        self.beta = [_spline(self.drho, k).to(DEVICE) for _, k in self.columns]


def _pick(tables, dx, element, x):
    """tables[element](x), element per value"""
    out = _eval(tables[0], dx, x)
    for e in range(1, len(tables)):
        out = torch.where(element == e, _eval(tables[e], dx, x), out)
    return out


def _pairs(x, lo, L, rc):
    """Directed pairs within rc of each other in a periodic box: i, j and the
    shift that takes x_j to the image next to x_i."""
    n = x.shape[0]
    nb = torch.tensor([int(float(l) / rc) for l in L], device=x.device)
    cell = torch.floor((x - lo) / L * nb).long().remainder(nb)
    flat = cell[:, 0] + nb[0] * (cell[:, 1] + nb[1] * cell[:, 2])
    order = torch.argsort(flat)
    count = torch.bincount(flat, minlength=int(nb.prod()))
    first = torch.cumsum(count, 0) - count
    most = int(count.max())
    me = torch.arange(n, device=x.device)
    I, J = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                c = (cell + torch.tensor([dx, dy, dz], device=x.device)).remainder(nb)
                c = c[:, 0] + nb[0] * (c[:, 1] + nb[1] * c[:, 2])
                f, k = first[c], count[c]
                for s in range(most):
                    i = me[k > s]
                    j = order[f[i] + s]
                    d = x[j] - x[i]
                    d = d - L * torch.round(d / L)
                    near = ((d * d).sum(1) < rc * rc) & (j != i)
                    I.append(i[near])
                    J.append(j[near])
    i, j = torch.cat(I), torch.cat(J)
    return i, j, -L * torch.round((x[j] - x[i]) / L)


def _philox(words, key):
    c = [np.asarray(w, dtype=np.uint64) for w in words]
    k = [np.uint64(v) for v in key]
    low = np.uint64(0xFFFFFFFF)
    for r in range(10):
        if r:
            k = [(k[0] + np.uint64(0x9E3779B9)) & low, (k[1] + np.uint64(0xBB67AE85)) & low]
        a, b = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(b >> np.uint64(32)) ^ c[1] ^ k[0], b & low, (a >> np.uint64(32)) ^ c[3] ^ k[1], a & low]
    return c


def _deviates(n, seed, step):
    """The fix's own deviates: Box-Muller on two Philox4x32-10 blocks."""
    def uniform(a, b):
        m = ((a >> np.uint64(5)) << np.uint64(26)) | (b >> np.uint64(6))
        return (m.astype(np.float64) + 0.5) * 2.0 ** -53

    i = np.arange(n, dtype=np.uint64)
    s = np.full(n, step, dtype=np.uint64)
    z = np.zeros(n, dtype=np.uint64)
    r, q = (_philox([i, s, z, z + np.uint64(w)], (seed, 0x9E3779B9)) for w in (0x45504847, 0x45504848))
    u = [uniform(r[0], r[1]), uniform(r[2], r[3]), uniform(q[0], q[1]), uniform(q[2], q[3])]
    ra, rb = np.sqrt(-2.0 * np.log(u[0])), np.sqrt(-2.0 * np.log(u[2]))
    t, w = 2.0 * np.pi * u[1], 2.0 * np.pi * u[3]
    return torch.from_numpy(np.stack([ra * np.cos(t), ra * np.sin(t), rb * np.cos(w)], 1)).to(DEVICE)


def _substeps(dt, h, c_min, r_min, k_max):
    r = dt * sum(1.0 / v / v for v in h) / c_min / r_min * k_max
    if not r > 0.4:
        return 1, dt
    n = max(1, int(dt / (0.4 * dt / r)))
    return n, dt / n


def _diffuse(T, dT, S, rhoC, kappa, flag, h, n, dt):
    """n substeps of the variable-kappa stencil on a (z, y, x) grid."""
    wall = flag == 2
    kp = kappa + torch.zeros_like(T)
    for _ in range(n):
        dd = torch.zeros_like(T)
        for axis, hh in ((2, h[0]), (1, h[1]), (0, h[2])):
            up, dn = wall.roll(-1, axis), wall.roll(1, axis)
            Tq, kq = torch.where(up, T, T.roll(-1, axis)), torch.where(up, kp, kp.roll(-1, axis))
            stay = dn & ~up
            Tp, kl = torch.where(stay, T, T.roll(1, axis)), torch.where(stay, kp, kp.roll(1, axis))
            dd = dd + (kq - kl) * (Tq - Tp) / (4.0 * hh * hh) + kp * (Tq + Tp - 2.0 * T) / (hh * hh)
        dd = torch.where(wall, torch.zeros_like(T), dd)
        T = torch.where(flag == 1, T + (dd + dT + S) / rhoC * dt, T).clamp(min=0.0)
    return T


class _Exact:
    """The fix's step on one system, FP64 and differentiable."""

    def __init__(self, case, seed):
        with tempfile.TemporaryDirectory() as folder:
            self.words, at = _system(case, seed, folder)
            self.tab = _Tables(self.words[16])
        self.case, self.dt, self.n = case, case["dt"], at.n
        self.x, self.v = _device(at.x), _device(at.v)
        self.f = _device(_start_force(at.n, seed))
        self.lo, self.L = _device(at.boxlo), _device(at.boxhi - at.boxlo)
        self.el = _device(at.type.astype(np.int64) - 1)
        self.mass = _device(at.mass)[self.el + 1][:, None]
        self.live = _device(at.mask == 1)
        self.g = (case["gx"], case["gy"], case["gz"])
        self.h = [float(l) / g for l, g in zip(self.L, self.g)]
        self.C, self.kappa = (torch.tensor(v, dtype=torch.float64, device=DEVICE) for v in (C_E, KAPPA))
        T = _grid_T(case, seed) if case["kind"] != "gradient" else np.full(math.prod(self.g), case["T_e"])
        self.T = _device(T).reshape(self.g[2], self.g[1], self.g[0])
        self.nsub, self.inner = _substeps(self.dt, self.h, C_E, RHO_E, KAPPA)
        self.count = 0

    def kick(self):
        dv = 0.5 * self.dt * W.FTM2V / self.mass * self.f
        self.v = self.v + torch.where(self.live[:, None], dv, torch.zeros_like(dv))

    def drift(self):
        self.x = self.x + torch.where(self.live[:, None], self.dt * self.v, torch.zeros_like(self.v))
        with torch.no_grad():  # into the box (an image, not a force)
            self.wrap = -self.L * torch.floor((self.x - self.lo) / self.L)

    def post_force(self, xi=None):
        """rho, beta, f_EPH and f_RNG of this step's positions"""
        tab, n = self.tab, self.n
        self.count += 1
        i, j, shift = _pairs(self.x.detach(), self.lo, self.L, tab.rc)
        e = self.x[j] + shift - self.x[i]
        r2 = (e * e).sum(1)
        if xi is None:
            xi = _deviates(n, int(self.words[3]), self.count)
        add = lambda rows, val: torch.zeros((n,) + val.shape[1:], dtype=torch.float64, device=DEVICE).index_add(0, rows, val)  # noqa: E731
        Hij = _pick(tab.rho, tab.dr2, self.el[j], r2)
        rho = torch.where(self.live, add(i, Hij), torch.zeros(n, dtype=torch.float64, device=DEVICE))
        Hij = Hij / r2
        Hji = _pick(tab.rho, tab.dr2, self.el[i], r2) / r2 if len(tab.rho) > 1 else Hij
        on = self.live & (rho > 0) & (rho <= tab.rho_max)
        one = torch.where(on, rho, torch.ones_like(rho))
        a = torch.where(on, _pick(tab.alpha, tab.drho, self.el, one) / one, torch.zeros_like(rho))
        beta = torch.where(self.live & (rho <= tab.rho_max), _pick(tab.beta, tab.drho, self.el, rho.clamp(max=tab.rho_max)),
                           torch.zeros_like(rho))
        w = a[:, None] * add(i, (Hij * (e * (self.v[i] - self.v[j])).sum(1))[:, None] * e)
        both = (self.live & (rho > 0))[i] & (self.live & (rho > 0))[j]
        i, j, e, Hij, Hji = i[both], j[both], e[both], Hij[both], Hji[both]

        def spread(y):
            return add(i, (a[i] * Hij * (e * y[i]).sum(1) - a[j] * Hji * (e * y[j]).sum(1))[:, None] * e)

        c = torch.floor((self.x.detach() - self.lo) / torch.tensor(self.h, device=DEVICE, dtype=torch.float64)).long()
        c = c.remainder(torch.tensor(self.g, device=DEVICE))
        self.cell = c[:, 0] + self.g[0] * (c[:, 1] + self.g[1] * c[:, 2])
        Te = self.T.reshape(-1)[self.cell]
        self.rho, self.beta = rho, beta
        self.f_eph = -spread(w)
        self.f_rng = math.sqrt(2.0 * W.BOLTZ / self.dt) * torch.sqrt(Te)[:, None] * spread(xi)
        self.f = self.f + self.f_eph + self.f_rng

    def end_of_step(self):
        dE = -((self.f_eph + self.f_rng) * self.v).sum(1) * self.dt
        dE = torch.where(self.live, dE, torch.zeros_like(dE))
        dV = math.prod(self.h)
        dT = torch.zeros(self.T.numel(), dtype=torch.float64, device=DEVICE).index_add(0, self.cell, dE / (dV * self.dt))
        flag = torch.ones_like(self.T, dtype=torch.int8)
        self.T = _diffuse(self.T, dT.reshape(self.T.shape), 0.0, RHO_E * self.C, self.kappa, flag, self.h, self.nsub, self.inner)
        return dE.sum()

    def step(self, pair=None):
        self.kick()
        self.drift()
        self.f = torch.zeros_like(self.f) if pair is None else pair(self)
        self.post_force()
        self.kick()
        return self.end_of_step()


class _ExactEam:
    """eam/alloy of one element on the setfl tables kept with the tests."""

    def __init__(self):
        tok = " ".join(lzma.decompress(open(NI_EAM, "rb").read()).decode().split("\n")[4:]).split()
        nrho, self.drho, nr, self.dr, self.rc = int(tok[0]), float(tok[1]), int(tok[2]), float(tok[3]), float(tok[4])
        v = np.array([float(t) for t in tok[9:9 + nrho + 2 * nr]])
        self.F, self.fr, self.z = (self._hermite(y) for y in (v[:nrho], v[nrho:nrho + nr], v[nrho + nr:]))
        self.rho_max = self.drho * (nrho - 1)

    @staticmethod
    def _hermite(y):
        s = np.empty_like(y)
        s[0], s[-1], s[1], s[-2] = y[1] - y[0], y[-1] - y[-2], 0.5 * (y[2] - y[0]), 0.5 * (y[-1] - y[-3])
        s[2:-2] = ((y[:-4] - y[4:]) + 8.0 * (y[3:-1] - y[1:-3])) / 12.0
        d = y[1:] - y[:-1]
        return _device(np.stack([y[:-1], s[:-1], 3.0 * d - 2.0 * s[:-1] - s[1:], s[:-1] + s[1:] - 2.0 * d], 1))

    @staticmethod
    def _at(c, q):
        m = q.long().clamp(0, c.shape[0] - 1)
        p = (q - m).clamp(max=1.0)
        k = c[m]
        return (k[:, 0] + p * (k[:, 1] + p * (k[:, 2] + p * k[:, 3])), k[:, 1] + p * (2.0 * k[:, 2] + 3.0 * p * k[:, 3]))

    def __call__(self, s):
        i, j, shift = _pairs(s.x, s.lo, s.L, self.rc)
        e = s.x[j] + shift - s.x[i]
        r = torch.sqrt((e * e).sum(1))
        f, df = self._at(self.fr, r / self.dr)
        rho = torch.zeros(s.n, dtype=torch.float64, device=DEVICE).index_add(0, i, f)
        F, dF = self._at(self.F, rho / self.drho)
        dF = dF / self.drho
        F = F + torch.where(rho > self.rho_max, dF * (rho - self.rho_max), torch.zeros_like(F))
        z, dz = self._at(self.z, r / self.dr)
        phi = z / r
        dEdr = (dF[i] + dF[j]) * df / self.dr + (dz / self.dr - phi) / r
        self.energy = float(F.sum() + 0.5 * phi.sum())
        return torch.zeros_like(s.x).index_add(0, i, (dEdr / r)[:, None] * e)


def _wrapped(s, start):
    """x as the fix leaves it: wrapped on steps where an atom had moved more
    than half the engine's skin since the last wrap (skin 1 A)."""
    if "since" not in s.__dict__:
        s.since = start
    if float(((s.x - s.since) ** 2).sum(1).max()) > 0.25:
        s.x = s.x + s.wrap
        s.since = s.x
    return s.x


def exact(case, seed):
    kind = case["kind"]
    if kind == "grid":
        a = _grid_arrays(case, seed)
        shape = (case["gz"], case["gy"], case["gx"])
        d = {k: _device(v).reshape(shape) for k, v in a.items()}
        h = [case["box"] / g for g in shape[::-1]]
        use = a["flag"] != 0
        use[0] = True
        n, dt = _substeps(case["dt"], h, a["C"][use].min(), a["rho"][use].min(), a["kappa"][use].max())
        T = _diffuse(d["T"], d["dT"], d["S"], d["rho"] * d["C"], d["kappa"], d["flag"], h, n, dt)
        return {"T": T.reshape(-1), "substeps": n}
    if kind == "batch":
        return [{k: v for k, v in exact(c, seed + 101 * r).items() if k in ("x", "v")}
                for r, c in enumerate(_replica_cases(case))]
    if 4 * case["nx"] * case["ny"] * case["nz"] > 600000:
        return None  # minutes in plain FP64
    s = _Exact(case, seed)
    if kind == "gradient":
        return _exact_gradient(s, case, seed)
    if kind == "hooks":
        s.f, s.count = _device(_start_force(s.n, seed)), 0
        s.post_force(_device(_host_xi(s.n, seed)) if case["xi"] == "host" else None)
        s.end_of_step()
        array = torch.cat([s.rho[:, None], s.beta[:, None], s.f_eph, s.f_rng], 1)
        return {"f": s.f, "array": array, "T": s.T.reshape(-1)}
    pair = _ExactEam() if kind == "md" else None
    start = s.x
    for _ in range(case["steps"]):
        s.kick()
        s.drift()
        _wrapped(s, start)
        s.f = torch.zeros_like(s.f) if pair is None else pair(s)
        s.post_force()
        s.kick()
        s.end_of_step()
    out = {"x": s.x, "v": s.v, "f": s.f, "T": s.T.reshape(-1)}
    if pair is not None:
        out["pair_energy"] = pair.energy
    return out


def _exact_gradient(s, case, seed):
    """The same gradient by reverse-mode differentiation of the FP64 steps."""
    r, b = s.tab.columns[0]
    b = b * (1.0 + 0.1 * torch.sin(torch.arange(64, dtype=torch.float64) / (4.0 + seed % 5)))
    leaves = [t.clone().requires_grad_(True) for t in (r, b, s.C, s.kappa)]
    s.tab.columns = [(leaves[0], leaves[1])]
    s.C, s.kappa = leaves[2], leaves[3]
    s.f = torch.zeros_like(s.f)  # an adjoint starts from a fresh context
    s.tab.build()
    E, T = [], []
    for _ in range(case["steps"]):
        E.append(s.step())
        T.append(s.T.mean())
    dE, dT = (_device(v) for v in _cotangents(case, seed))
    E, T = torch.stack(E), torch.stack(T)
    g = torch.autograd.grad((E * dE).sum() + (T * dT).sum(), leaves)
    return {"rho_knots": g[0], "beta_knots": g[1], "C_e": float(g[2]), "kappa_e": float(g[3]), "E": E.detach(), "T": T.detach()}
