"""The work a user of the library has it do, as cases that can be timed and compared.

A pass takes the state from the host's page-locked arrays through the public entry points and
back, as the time loop of a host program does: upload, some steps (or a recorded window and its
reverse sweep, or a batch of simulations), download.  One case is a block on its own, the PPE
solve on a matrix the caller holds in device memory.

Sizes and physical parameters are those of the generators in vebisph_gb300/cases.py and of the
benchmark.  States are mid-flow, not the generators' states of rest: a velocity with a smooth
seeded disturbance and a conformation tensor with distinct eigenvalues, which is what every step
but a run's first few works on (at rest the pressure equation has no right-hand side, and at
A = I the reference's log-conformation update divides by 1e-10).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from vebisph_gb300 import abi, cases
from vebisph_gb300.solver import Adjoint, BatchSolver, StepSolver, VebiError

PAIRS = 44.0  # neighbours of a particle inside the support 3h at h = 1.3 dx


def listed():
    return [
        # the smallest run there is: the 40 x 40 channel, ten steps of a time loop; all launches and latency
        {"name": "channel_40_fp64", "kind": "step", "geometry": "channel", "n": 40, "precision": "fp64",
         "precond": "none", "steps": 10, "dump": False},
        # the input deck the reference ships (10,102 particles, PTT, two walls and a periodic pair) with a
        # dump-time step at the end (vorticity)
        {"name": "deck_10k_fp64", "kind": "step", "geometry": "deck", "n": 101, "precision": "fp64",
         "precond": "none", "steps": 4, "dump": True},
        # the generator's free-surface deck: open domain, Jacobi BiCGSTAB, PTT, velocity-dependent shifting
        {"name": "free_surface_75_fp64", "kind": "step", "geometry": "free_surface", "n": 75, "precision": "fp64",
         "precond": "none", "steps": 4, "dump": False},
        # a production-size run on the reference's solver
        {"name": "cylinder_100k_fp64", "kind": "step", "geometry": "cylinder", "n": 100_000, "precision": "fp64",
         "precond": "none", "steps": 1, "dump": False},
        # the headline benchmark's step: 4M particles, FP64, the reference's solver to its iteration cap
        {"name": "cylinder_4m_fp64", "kind": "step", "geometry": "cylinder", "n": 4_000_000, "precision": "fp64",
         "precond": "none", "steps": 1, "dump": False},
        # the same step with the multigrid preconditioner, in both precisions
        {"name": "cylinder_4m_fp64_mg", "kind": "step", "geometry": "cylinder", "n": 4_000_000, "precision": "fp64",
         "precond": "multigrid", "steps": 1, "dump": False},
        {"name": "cylinder_4m_mixed_mg", "kind": "step", "geometry": "cylinder", "n": 4_000_000,
         "precision": "mixed", "precond": "multigrid", "steps": 1, "dump": False},
        # one simulation of a parameter study on its own, in the mode such a study runs in
        {"name": "cylinder_20k_mixed_mg", "kind": "step", "geometry": "cylinder", "n": 20_000,
         "precision": "mixed", "precond": "multigrid", "steps": 4, "dump": False},
        # a parameter study: 24 independent channels and cylinders of 4k to 256k particles advanced together
        {"name": "batch_24_mixed_mg", "kind": "batch", "instances": 24, "lo": 4_000, "hi": 256_000,
         "precision": "mixed", "precond": "multigrid", "steps": 1},
        # gradients on the heated cavity of the benchmark (1M particles): record a window, reverse it
        {"name": "adjoint_cavity_1024_fp64", "kind": "adjoint", "n": 1024, "precision": "fp64",
         "precond": "multigrid", "const_mod": 2, "steps": 2, "checkpoint": 2},
        # the same at the size of an optimisation study, in mixed precision, with a recomputed segment
        {"name": "adjoint_cavity_96_mixed", "kind": "adjoint", "n": 96, "precision": "mixed",
         "precond": "multigrid", "const_mod": 2, "steps": 4, "checkpoint": 2},
        # the PPE solve alone, for a caller that may not allocate: the matrix is the caller's
        {"name": "ppe_noalloc_128", "kind": "ppe", "nx": 128, "ny": 128, "closed": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "batch", "adjoint", "ppe"])
    if kind == "ppe":
        nx = _log(rng, 24, 256)
        return {"kind": "ppe", "nx": nx, "ny": _log(rng, 24, 65536 // nx),
                "closed": rng.random() < 0.7}
    if kind == "adjoint":
        precision = rng.choice(["fp64", "mixed"])
        return {"kind": "adjoint", "n": _log(rng, 20, 400), "precision": precision, "precond": "multigrid",
                "const_mod": rng.choice([1, 2]), "steps": rng.randint(2, 4), "checkpoint": rng.randint(1, 3)}
    if kind == "batch":
        return {"kind": "batch", "instances": rng.randint(3, 24), "lo": 4_000, "hi": _log(rng, 16_000, 256_000),
                "precision": rng.choice(["mixed", "mixed", "fp64"]), "precond": rng.choice(["multigrid", "none"]),
                "steps": 1}
    precision, precond = rng.choice([("fp64", "none"), ("fp64", "multigrid"), ("mixed", "multigrid"),
                                     ("mixed", "none")])
    geometry = rng.choice(["channel", "cylinder", "cavity", "free_surface", "dam_break"])
    fluid = _log(rng, 1_600, 1_000_000 if precond == "multigrid" else 130_000)
    if geometry in ("free_surface", "dam_break"):
        fluid = _log(rng, 1_600, 130_000)
    n = {"channel": math.sqrt(fluid), "cavity": math.sqrt(fluid), "cylinder": max(fluid, 4_000),
         "free_surface": math.sqrt(2.0 * fluid), "dam_break": math.sqrt(0.5 * fluid)}[geometry]
    return {"kind": "step", "geometry": geometry, "n": int(round(n)), "precision": precision, "precond": precond,
            "steps": 1 if fluid > 60_000 else rng.randint(1, 4), "dump": rng.random() < 0.2}


# ------------------------------------------------------------------------------- inputs
def _modes(rng, x, y, lx, ly, k=4):
    """A smooth seeded field of order one, zero on y = 0 and y = ly and periodic in x over lx."""
    f = np.zeros_like(x)
    for _ in range(k):
        a, mx, my, ph = rng.normal(), int(rng.integers(1, 5)), int(rng.integers(1, 5)), rng.uniform(0, 2 * math.pi)
        f += a * np.sin(2 * math.pi * mx * x / lx + ph) * np.sin(math.pi * my * y / ly)
    return f / math.sqrt(k)


def _mid_flow(c, geometry, seed):
    """Velocity and conformation of a developed flow with a disturbance, into the case."""
    rng = np.random.default_rng(seed + 1000)
    nb = c.nbS
    x0, y0 = c.b_node.min(axis=0)
    lx, ly = c.b_node.max(axis=0) - c.b_node.min(axis=0)
    x, y = c.r[:, 0] - x0, c.r[:, 1] - y0
    fu, fv, ft = (_modes(rng, x, y, lx, ly) for _ in range(3))
    wi = c.El * math.sqrt(c.Ra / c.Pr)
    if geometry in ("channel", "cylinder"):  # the steady Oldroyd-B channel
        um = 1.0 if geometry == "channel" else 1.5
        u = um * 4.0 * (y / ly) * (1.0 - y / ly)
        shear = wi * um * 4.0 / ly * (1.0 - 2.0 * y / ly)
        c.u[nb:, 0] = (u + 0.02 * fu)[nb:]
        c.u[nb:, 1] = (0.02 * fv)[nb:]
        txx, txy, tyy = 2.0 * shear * shear + 0.3 + 0.05 * ft, shear, np.zeros_like(x)
    else:
        c.u[nb:, 0], c.u[nb:, 1] = (0.05 * fu)[nb:], (0.05 * fv)[nb:]
        txx, txy, tyy = 0.6 + 0.1 * ft, 0.2 + 0.05 * fu, 0.1 + 0.02 * fv
        c.theta[nb:] += 0.01 * ft[nb:]
    if c.const_mod != 1:
        c.tau = np.stack([txx, txy, txy, tyy], 1)
        c.trace_conf = 2.0 + txx + tyy
    return c


def _case(geometry, n, seed, const_mod=2):
    if geometry == "channel":
        c = cases.poiseuille(n, seed=seed)
    elif geometry == "cylinder":
        c = cases.cylinder(float(n), Wi=0.6, seed=seed)
    elif geometry == "cavity":
        c = cases.cavity(n, seed=seed)
    elif geometry == "free_surface":
        c = cases.free_surface_periodic(n, seed=seed)
    elif geometry == "dam_break":
        c = cases.dam_break(n, seed=seed)
    else:  # the shipped deck, its lattice disturbed as a run's is after some steps
        c = cases.rayleigh_benard_deck()
        c.r[c.nbS:] += np.random.default_rng(seed).uniform(-0.01 * c.dx, 0.01 * c.dx, (c.npfb - c.nbS, 2))
    if const_mod == 1:
        c.const_mod = 1
    return _mid_flow(c, geometry, seed)


def _set_mode(c, case):
    c.ppe_precond = abi.PRECOND_MULTIGRID if case["precond"] == "multigrid" else abi.PRECOND_NONE
    return abi.PREC_MIXED if case["precision"] == "mixed" else abi.PREC_FP64


def _pinned(shape, dtype=np.float64):
    t = {np.float64: torch.float64, np.int32: torch.int32, np.uint8: torch.uint8}[dtype]
    return torch.zeros(shape, dtype=t, pin_memory=True).numpy()


FIELDS = (("r", 2), ("u", 2), ("tau", 4), ("theta", 1), ("p", 1), ("vort", 1), ("a_out", 1), ("trace_conf", 1))


class _Host:
    """The host program's arrays of several simulations, one page-locked array per field: the state it
    passes in (inp) and the state it gets back (out)."""

    def __init__(self, cs):
        self.n = [c.npfb for c in cs]
        self.at = np.concatenate([[0], np.cumsum(self.n)]).astype(int)
        tot = int(self.at[-1])
        self.inp = {k: _pinned(m * tot) for k, m in FIELDS if k not in ("p", "vort", "a_out")}
        self.inp["inbin"] = _pinned(tot, np.uint8)
        self.out = {k: _pinned(m * tot) for k, m in FIELDS}
        self.out["n_surf"] = _pinned(tot, np.int32)
        self.out["inbin"] = _pinned(tot, np.uint8)
        for i, c in enumerate(cs):
            f = c.fortran_planes()
            for k in ("r", "u", "tau", "theta", "trace_conf"):
                self.part(self.inp, k, i)[:] = np.asarray(f[k]).reshape(-1)

    def part(self, side, k, i):
        m = dict(FIELDS).get(k, 1)
        return side[k][m * self.at[i]:m * self.at[i + 1]]

    def upload(self, solver, i):
        a = [self.part(self.inp, k, i) for k in ("r", "u", "tau", "theta", "trace_conf", "inbin")]
        solver.upload(*a, self.n[i])

    def download(self, solver, i):
        dp = [self.part(self.out, k, i).ctypes.data_as(C.POINTER(C.c_double)) for k, _ in FIELDS[:4]]
        dp += [self.part(self.out, k, i).ctypes.data_as(C.POINTER(C.c_double)) for k, _ in FIELDS[4:]]
        st = solver.lib.vebi_download_state(
            solver.h, *dp, self.part(self.out, "n_surf", i).ctypes.data_as(C.POINTER(C.c_int32)),
            self.part(self.out, "inbin", i).ctypes.data_as(C.POINTER(C.c_uint8)), self.n[i])
        if st:
            raise VebiError(st, "vebi_download_state", solver.lib.vebi_last_error().decode())


def _ppe_system(case, seed):
    """The pressure matrix of a doubly periodic jittered nx x ny lattice (quintic-spline Morris weights, all
    pairs inside 3h), in the ELL layout of the step; closed: zero row sums and a mean-free right-hand side,
    open: the lattice's last row of particles is a free surface (diagonal 1e30)."""
    nx, ny = case["nx"], case["ny"]
    n = nx * ny
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)
    h = 1.3
    i = torch.arange(n, device=dev)
    ix, iy = i // ny, i % ny
    jit = (torch.rand(n, 2, generator=g, device=dev, dtype=torch.float64) - 0.5) * 0.02
    cols, vals = [], []
    for dx in range(-4, 5):
        for dy in range(-4, 5):
            if (dx == 0 and dy == 0) or dx * dx + dy * dy > 17:
                continue
            j = ((ix + dx) % nx) * ny + (iy + dy) % ny
            rx = -float(dx) + jit[:, 0] - jit[j, 0]
            ry = -float(dy) + jit[:, 1] - jit[j, 1]
            q = torch.sqrt(rx * rx + ry * ry) / h
            f = sum(w * torch.clamp(k - q, min=0.0) ** 4 for w, k in ((-5.0, 3.0), (30.0, 2.0), (-75.0, 1.0)))
            cols.append(j)
            vals.append(torch.where(q <= 3.0, 2.0 * f * 7.0 / 478.0 / math.pi / h ** 3 / (q * h), 0.0))
    col, val = torch.stack(cols), -torch.stack(vals)
    keep = val != 0.0
    order = torch.argsort((~keep).to(torch.int8), dim=0, stable=True)
    cnt = keep.sum(0).to(torch.int32)
    width = int(cnt.max())
    col = torch.gather(col, 0, order)[:width].to(torch.int32).contiguous()
    val = torch.gather(val, 0, order)[:width].contiguous()
    val[torch.arange(width, device=dev)[:, None] >= cnt[None, :]] = 0.0
    diag = -val.sum(0)
    rhs = torch.randn(n, generator=g, device=dev, dtype=torch.float64)
    for k in range(1, 4):
        a = torch.randn(2, generator=g, device=dev, dtype=torch.float64)
        rhs += 3.0 * a[0] * torch.sin(2 * math.pi * k * ix / nx + a[1]) * torch.cos(2 * math.pi * k * iy / ny)
    if case["closed"]:
        rhs -= rhs.mean()
    else:
        diag[iy == ny - 1] = 1.0e30
    return {"cnt": cnt, "col": col, "val": val, "diag": diag.contiguous(), "rhs": rhs, "n": n}


def prepare(case, seed):
    if case["kind"] == "ppe":
        s = _ppe_system(case, seed)
        s |= {"kind": "ppe", "closed": int(case["closed"]), "x": torch.zeros_like(s["rhs"]), "lib": abi.load_library()}
        return s
    if case["kind"] == "batch":
        # the benchmark's sweep: alternating channels and cylinders, log-uniform sizes, Wi and beta spread
        cs = cases.batch_sweep(case["instances"], seed=seed % 100_000, lo=float(case["lo"]), hi=float(case["hi"]))
        # every run of a case costs the same: the sizes are the case's, the rest is the seed's
        sizes = np.exp(np.linspace(math.log(case["lo"]), math.log(case["hi"]), case["instances"]))
        for k, c in enumerate(cs):
            wi, beta = c.El * math.sqrt(c.Ra / c.Pr), c.beta
            cs[k] = _mid_flow(cases.poiseuille(int(round(math.sqrt(sizes[k]))), seed=seed + k, Wi=wi, beta=beta) if k % 2 == 0
                              else cases.cylinder(float(sizes[k]), Wi=wi, beta=beta, seed=seed + k),
                              "channel" if k % 2 == 0 else "cylinder", seed + k)
            prec = _set_mode(cs[k], case)
        b = BatchSolver(cs, precision=prec)
        b.set_solver_grid(4)  # what the autotuner picks for the sweep
        return {"kind": "batch", "batch": b, "host": _Host(cs), "steps": case["steps"]}
    if case["kind"] == "adjoint":
        c = _case("cavity", case["n"], seed, case["const_mod"])
        solver = StepSolver(c, precision=_set_mode(c, case))
        adj = Adjoint(solver, max_steps=case["steps"], checkpoint_every=case["checkpoint"])
        x, y = c.r[:, 0], c.r[:, 1]
        rng = np.random.default_rng(seed + 2000)
        n = c.npfb
        seeds = {"seed_u": np.stack([_modes(rng, x, y, 1.0, 1.0), _modes(rng, x, y, 1.0, 1.0)]) / n,
                 "seed_theta": _modes(rng, x, y, 1.0, 1.0) / n,
                 "seed_tau": np.stack([_modes(rng, x, y, 1.0, 1.0) for _ in range(4)]) / n}
        return {"kind": "adjoint", "solver": solver, "adjoint": adj, "host": _Host([c]), "seeds": seeds,
                "steps": case["steps"]}
    c = _case(case["geometry"], case["n"], seed)
    solver = StepSolver(c, precision=_set_mode(c, case))
    return {"kind": "step", "solver": solver, "host": _Host([c]), "steps": case["steps"], "dump": case["dump"]}


# ------------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "ppe":
        s = state
        st = s["lib"].vebi_ppe_solve_noalloc(
            s["cnt"].data_ptr(), s["col"].data_ptr(), s["val"].data_ptr(), s["diag"].data_ptr(), s["rhs"].data_ptr(),
            s["x"].data_ptr(), s["n"], s["n"], s["closed"], 1.0e-8, 1000,
            C.c_void_p(torch.cuda.current_stream().cuda_stream), None, None)
        if st:
            raise VebiError(st, "vebi_ppe_solve_noalloc", s["lib"].vebi_last_error().decode())
        return s["x"]
    host = state["host"]
    if kind == "batch":
        b = state["batch"]
        for i, inst in enumerate(b.instances):
            host.upload(inst, i)
        b.step(state["steps"])
        for i, inst in enumerate(b.instances):
            host.download(inst, i)
        return host.out
    solver = state["solver"]
    host.upload(solver, 0)
    if kind == "adjoint":
        state["adjoint"].record(state["steps"])
        g = state["adjoint"].reverse(**state["seeds"])
        return {k: g[k] for k in ("u", "theta", "tau", "wi")}
    for k in range(state["steps"]):
        solver.step(secondary=state["dump"] and k + 1 == state["steps"])
    host.download(solver, 0)
    return host.out


# ------------------------------------------------------------------------------- what a pass needs
def _particles(case):
    n = case["n"]
    g = case["geometry"]
    return {"channel": n * n, "cavity": n * n, "deck": n * n, "cylinder": n, "free_surface": n * n / 2,
            "dam_break": 2 * n * n}[g]


def _iterations(n, precond):
    """PPE iterations of a step: the multigrid solver's hardly grow with the size; the reference's grow with
    the lattice's edge, up to the cap."""
    return 14.0 + 1.0 * math.log10(max(n, 10.0) / 1e4) if precond == "multigrid" else min(1001.0, 1.6 * math.sqrt(n))


def _step_flops(n, precond):
    # pair operators: distance, kernel and its derivative, weights, correction, shifting, six gradients, stress
    # and viscous sums, right-hand side, pressure gradient; per iteration two matrix products and the recurrences
    pairs = 190.0 * PAIRS * n
    it = 2.0 * (2.0 * (PAIRS + 1.0)) + 26.0
    return pairs + 300.0 * n + _iterations(n, precond) * it * n


def work(case):
    if case["kind"] == "ppe":
        n = case["nx"] * case["ny"]
        return {"bytes": (12.0 * PAIRS + 28.0) * n,
                "flops": 0.6 * _iterations(n, "none") * (4.0 * (PAIRS + 1.0) + 26.0) * n}
    if case["kind"] == "batch":
        sizes = np.exp(np.linspace(math.log(case["lo"]), math.log(case["hi"]), case["instances"]))
        n = float(sizes.sum())
        flops = case["steps"] * sum(_step_flops(float(m), case["precond"]) for m in sizes)
    elif case["kind"] == "adjoint":
        n = float(case["n"]) ** 2
        # a recorded step, its recomputation without the solve, and a reverse step with a transposed solve
        flops = case["steps"] * 3.0 * _step_flops(n, case["precond"])
        return {"bytes": (81.0 + 112.0) * n, "flops": flops}
    else:
        n = float(_particles(case))
        flops = case["steps"] * _step_flops(n, case["precond"])
    return {"bytes": (81.0 + 109.0) * n, "flops": flops}  # the state in, the fields out


# ------------------------------------------------------------------------------- the exact answer
def exact(case, seed):
    """The PPE block's system has a solution to compare with; it is solved here to 64-bit rounding by conjugate
    gradients (the matrix is symmetric).  A whole step has none: its pressure is the iterate at which
    BiCGSTAB's residual test stops (or the iteration cap), and everything after it follows."""
    if case["kind"] != "ppe":
        return None
    s = _ppe_system(case, seed)
    col, closed = s["col"].long(), bool(case["closed"])
    free = (s["diag"] != 1.0e30).to(torch.float64)  # a free-surface row's value is rhs / 1e30
    val, diag, b = -s["val"], torch.where(free == 0.0, 1.0, -s["diag"]), -s["rhs"]

    def mul(x):  # the matrix is negative (semi)definite on the other rows
        return free * (diag * x + (val * x[col]).sum(0))

    x = torch.zeros_like(b)
    for _ in range(3):  # restarted on the true residual
        r = free * (b - mul(x))
        if closed:
            r = r - r.mean()
        z = r / diag
        p, rz = z, torch.dot(r, z)
        first = float(rz)
        for _ in range(4000):
            if float(rz) <= 1e-28 * first or first == 0.0:
                break
            ap = mul(p)
            a = rz / torch.dot(p, ap)
            x = x + a * p
            r = r - a * ap
            if closed:
                r = r - r.mean()
            z = r / diag
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
        if closed:
            x = x - x.mean()
    x = torch.where(free == 0.0, s["rhs"] / 1.0e30, x)
    return x
