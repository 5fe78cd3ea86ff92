"""Performance cases: the batch solves this package is used for.

Each case is one call of a public entry point (``Solver.solve``,
``HeteroSolver.solve``, ``AdjointIntegrator``) on seeded inputs of a named
kind, from a small parameter sweep that is bound by launch latency to the
ensembles of ``bench.py``.  ``exact`` gives the same outputs from plain torch
in FP64: extrapolated modified midpoint for non-stiff systems, extrapolated
linearly implicit Euler for stiff ones, and the fixed-step method itself
where the step is part of the definition (the cable).
"""

import functools
import math

import numpy as np
import torch

from cubie_b200 import Solver, create_ODE_system
from cubie_b200.adjoint import AdjointIntegrator
from cubie_b200.hetero import HeteroSolver
from cubie_b200.interpolator import ArrayInterpolator

LORENZ = ["dx = sigma * (y - x)", "dy = x * (rho - z) - y", "dz = x * y - beta * z"]
VDP = ["dx = y", "dy = mu * (1 - x**2) * y - x"]
FHN = ["dV = V - V**3 / 3 - w + I", "dw = (V + a - b * w) / tau"]
ROBERTSON = ["dy1 = -k1 * y1 + k3 * y2 * y3", "dy2 = k1 * y1 - k3 * y2 * y3 - k2 * y2**2", "dy3 = k2 * y2**2"]
DRIVEN = ["dx = v", "dv = -k * x - c * v + F", "E = 0.5 * v**2 + 0.5 * k * x**2"]
SIGMA, BETA = 10.0, 8.0 / 3.0


def listed():
    return [
        # a notebook-sized sweep: arrays in, arrays out, the defaults' FP32;
        # latency and launches count
        dict(name="lorenz_sweep_96", kind="lorenz", runs=96, precision="float32", algorithm="dormand-prince-54",
             horizon=2.0, host=True),
        # saved trajectories and summaries of an ordinary ensemble
        dict(name="lorenz_rows_4096", kind="lorenz_rows", runs=4096, rows=200, precision="mixed"),
        # double precision at a tight tolerance, an odd number of runs
        dict(name="lorenz_f64_50021", kind="lorenz", runs=50021, precision="float64", algorithm="tsit5",
             horizon=2.0, host=False),
        # a stiff ensemble of ordinary size, per-run horizons, data on the GPU
        dict(name="vdp_ros3p_20011", kind="vdp", runs=20011, algorithm="ros3p", linear="direct", precision="mixed",
             host=False),
        # the benchmark's stiff ensemble from pinned host memory and back
        dict(name="vdp_ros3p_1048576", kind="vdp", runs=1 << 20, algorithm="ros3p", linear="direct",
             precision="mixed", host=True, spread=True),
        # fully implicit Radau IIA with matrix-free GMRES
        dict(name="vdp_radau_65536", kind="vdp", runs=65536, algorithm="radau", linear="gmres", precision="mixed",
             host=False),
        # sampled driver input, observables and times saved, default linear solver
        dict(name="driven_sdirk_30001", kind="driven", runs=30001, rows=50),
        # a large system, one warp per run: the benchmark's 256-state cable
        dict(name="cable64_1536", kind="cable", compartments=64, runs=1536, horizon=2.5),
        # a smaller cable, many runs
        dict(name="cable19_5003", kind="cable", compartments=19, runs=5003, horizon=2.5),
        # gradient fitting: forward and discrete adjoint, explicit tableau
        dict(name="fhn_fit_131072", kind="fhn_fit", runs=131072, horizon=60),
        # and through a Rosenbrock method
        dict(name="vdp_fit_8191", kind="vdp_fit", runs=8191, horizon=6),
        # three systems with their own horizons and tolerances in one launch
        dict(name="mixed_batch_150000", kind="mixed", runs=150000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lorenz", "lorenz", "lorenz_rows", "vdp", "vdp", "vdp", "driven", "cable", "cable", "fhn_fit",
                       "vdp_fit", "mixed"])
    if kind == "lorenz":
        return dict(kind=kind, runs=_log_int(rng, 32, 200000), precision=rng.choice(["float32", "mixed", "float64"]),
                    algorithm=rng.choice(["dormand-prince-54", "tsit5"]), horizon=round(rng.uniform(0.5, 2.0), 3),
                    host=rng.random() < 0.5)
    if kind == "lorenz_rows":
        return dict(kind=kind, runs=_log_int(rng, 100, 60000), rows=rng.randint(20, 200),
                    precision=rng.choice(["float32", "mixed", "float64"]))
    if kind == "vdp":
        algorithm, linear = rng.choice([("ros3p", "direct"), ("ros3p", "direct"), ("ros3p", "gmres"),
                                        ("radau", "direct"), ("radau", "gmres")])
        precision = rng.choice(["mixed", "mixed", "float64"])
        return dict(kind=kind, runs=_log_int(rng, 200, 500000 if algorithm == "ros3p" else 100000),
                    algorithm=algorithm, linear=linear, precision=precision, host=rng.random() < 0.3)
    if kind == "driven":
        return dict(kind=kind, runs=_log_int(rng, 300, 100000), rows=rng.randint(10, 60))
    if kind == "cable":
        return dict(kind=kind, compartments=rng.randint(16, 64), runs=_log_int(rng, 100, 3000),
                    horizon=0.5 * rng.randint(2, 5))
    if kind == "fhn_fit":
        return dict(kind=kind, runs=_log_int(rng, 500, 131072), horizon=rng.randint(20, 60))
    if kind == "vdp_fit":
        return dict(kind=kind, runs=_log_int(rng, 200, 30000), horizon=rng.randint(3, 6))
    return dict(kind=kind, runs=_log_int(rng, 3000, 150000))


# ---------------------------------------------------------------------------
# inputs (host, FP64) and solvers
# ---------------------------------------------------------------------------
def _released(rng, n):
    """Van der Pol runs let go on either slow branch near its fold: one
    relaxation jump early in the run, the next after about 0.8 mu."""
    side = np.where(rng.random(n) < 0.5, -1.0, 1.0)
    return np.stack([side * rng.uniform(1.1, 1.6, n), rng.uniform(-0.5, 0.5, n)])


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    n = case["runs"]
    kind = case["kind"]
    if kind in ("lorenz", "lorenz_rows"):
        return dict(x0=rng.uniform(-10.0, 10.0, (3, n)), p=rng.uniform(20.0, 35.0, (1, n)))
    if kind == "vdp":
        mu = 10.0 ** rng.uniform(0.0, 3.0, n)
        if case.get("spread"):
            # the benchmark's draw: any phase, a few relaxation jumps a run,
            # some runs still inside one when they end
            return dict(x0=rng.uniform(-2.0, 2.0, (2, n)), p=mu[None, :], durations=2.0 * mu)
        return dict(x0=_released(rng, n), p=mu[None, :], durations=mu * rng.uniform(0.5, 0.7, n))
    if kind == "driven":
        phase = rng.uniform(0.0, 2.0 * np.pi)
        s = np.sin(2.0 * np.pi * np.arange(41) / 40 + phase) + 0.5 * np.sin(6.0 * np.pi * np.arange(41) / 40)
        s[-1] = s[0]
        return dict(x0=rng.uniform(-1.0, 1.0, (2, n)),
                    p=np.stack([rng.uniform(0.5, 4.0, n), rng.uniform(0.1, 0.5, n)]),
                    samples=s.astype(np.float32))
    if kind == "cable":
        nc = case["compartments"]
        rest = np.repeat([-65.0, 0.05, 0.6, 0.32], nc)[:, None]
        scale = np.repeat([0.5, 0.005, 0.005, 0.005], nc)[:, None]
        s = np.where(np.arange(51) < 25, 10.0, 0.0)
        s[-1] = s[0]
        return dict(x0=rest + scale * rng.normal(0.0, 1.0, (4 * nc, n)),
                    p=np.stack([rng.uniform(80, 160, n), rng.uniform(20, 50, n), rng.uniform(0.1, 1.0, n)]),
                    samples=s.astype(np.float32))
    if kind == "fhn_fit":
        # on the spiking side of the excitability threshold
        return dict(x0=np.stack([rng.uniform(1.0, 2.0, n), rng.uniform(-0.5, 0.5, n)]),
                    p=np.stack([rng.uniform(0.6, 0.8, n), rng.uniform(0.7, 0.9, n), rng.uniform(8.0, 13.0, n),
                                rng.uniform(0.5, 0.7, n)]),
                    target=rng.uniform(-1.0, 1.0, (case["horizon"] + 1, n)))
    if kind == "vdp_fit":
        return dict(x0=np.stack([rng.uniform(1.0, 2.0, n), rng.uniform(-1.0, 1.0, n)]), p=rng.uniform(0.5, 3.0, (1, n)),
                    target=rng.uniform(-2.0, 2.0, (case["horizon"] + 1, n)))
    m = n // 3
    fams = [dict(x0=rng.uniform(-10.0, 10.0, (3, m)), p=rng.uniform(20.0, 35.0, (1, m)),
                 durations=10.0 ** rng.uniform(-0.7, 0.3, m))]
    mu = 10.0 ** rng.uniform(0.0, 3.0, m)
    fams.append(dict(x0=_released(rng, m), p=mu[None, :], durations=mu * rng.uniform(0.5, 0.7, m)))
    fams.append(dict(x0=np.tile([[1.0], [0.0], [0.0]], (1, m)),
                     p=np.stack([0.04 * rng.uniform(0.5, 2, m), 3e7 * rng.uniform(0.5, 2, m),
                                 1e4 * rng.uniform(0.5, 2, m)]),
                     durations=10.0 ** rng.uniform(0.0, 3.0, m)))
    for f in fams:
        f["tol_scale"] = 10.0 ** rng.uniform(-3.0, 0.0, m)
    return dict(families=fams)


def _cable_equations(nc):
    V = [f"V{j:02d}" for j in range(nc)]
    eqs = []
    for j, v in enumerate(V):
        left, right = V[max(j - 1, 0)], V[min(j + 1, nc - 1)]
        eqs.append(f"d{v} = {'I + ' if j == 0 else ''}gc * ({left} - 2 * {v} + {right})"
                   f" - gNa * m{j:02d}**3 * h{j:02d} * ({v} - 50.0) - gK * n{j:02d}**4 * ({v} + 77.0)"
                   f" - 0.3 * ({v} + 54.4)")
    # x / (1 - exp(-x)) by its series near x = 0, as FP32 needs it
    def gate(v, v0):
        x = f"(({v} + {v0}) / 10.0)"
        return f"({x} / (1 - exp(-{x})) if abs({x}) > 0.1 else 1 + {x} / 2 + {x}**2 / 12)"

    eqs += [f"dm{j:02d} = {gate(v, 40.0)} * (1 - m{j:02d})"
            f" - 4.0 * exp(-({v} + 65.0) / 18.0) * m{j:02d}" for j, v in enumerate(V)]
    eqs += [f"dh{j:02d} = 0.07 * exp(-({v} + 65.0) / 20.0) * (1 - h{j:02d})"
            f" - 1.0 / (1 + exp(-({v} + 35.0) / 10.0)) * h{j:02d}" for j, v in enumerate(V)]
    eqs += [f"dn{j:02d} = 0.1 * {gate(v, 55.0)} * (1 - n{j:02d})"
            f" - 0.125 * exp(-({v} + 65.0) / 80.0) * n{j:02d}" for j, v in enumerate(V)]
    states = [*V, *(f"{g}{j:02d}" for g in "mhn" for j in range(nc))]
    return eqs, states


def _precision(case):
    name = case.get("precision", "mixed")
    return (np.float64 if name == "float64" else np.float32), name == "mixed"


@functools.lru_cache(maxsize=None)
def _system(name, double, nc=0):
    p = np.float64 if double else np.float32
    if name == "lorenz":
        return create_ODE_system(LORENZ, states=["x", "y", "z"], parameters=["rho"],
                                 constants={"sigma": SIGMA, "beta": BETA}, precision=p)
    if name == "vdp":
        return create_ODE_system(VDP, states=["x", "y"], parameters=["mu"], precision=p)
    if name == "fhn":
        return create_ODE_system(FHN, states=["V", "w"], parameters=["a", "b", "tau", "I"], precision=p)
    if name == "robertson":
        return create_ODE_system(ROBERTSON, states=["y1", "y2", "y3"], parameters=["k1", "k2", "k3"], precision=p)
    if name == "driven":
        return create_ODE_system(DRIVEN, states=["x", "v"], parameters=["k", "c"], observables=["E"], drivers=["F"],
                                 precision=p)
    eqs, states = _cable_equations(nc)
    return create_ODE_system(eqs, states=states, parameters=["gNa", "gK", "gc"], drivers=["I"], precision=p)


@functools.lru_cache(maxsize=None)
def _solver(kind, algorithm, linear, precision, nc):
    """The solver a program keeps: one per configuration, whatever the inputs."""
    double, mixed = precision == "float64", precision == "mixed"
    if kind == "lorenz":
        tol = dict(rtol=1e-9, atol=1e-11) if double else dict(rtol=1e-6, atol=1e-8)
        return Solver(_system("lorenz", double), algorithm=algorithm, mixed_precision=mixed, output_types=["state"],
                      **tol)
    if kind == "lorenz_rows":
        tol = dict(rtol=1e-9, atol=1e-11) if double else dict(rtol=1e-6, atol=1e-8)
        return Solver(_system("lorenz", double), algorithm="dormand-prince-54", mixed_precision=mixed,
                      output_types=["state", "mean", "max"], save_every=0.01, summarise_every=0.1,
                      sample_summaries_every=0.01, **tol)
    if kind == "vdp":
        return Solver(_system("vdp", double), algorithm=algorithm, linear_correction_type=linear,
                      preconditioner_type=None, mixed_precision=mixed, rtol=1e-6, atol=1e-6, output_types=["state"],
                      save_variables=["x"])
    if kind == "driven":
        return Solver(_system("driven", False), algorithm="l_stable_sdirk_4", rtol=1e-4, atol=1e-4,
                      save_every=0.5, output_types=["state", "observables", "time"])
    if kind == "cable":
        return Solver(_system("cable", False, nc), algorithm="l_stable_dirk_3", linear_correction_type="bicgstab",
                      layout="auto", dt=0.03125, rtol=1e-4, atol=1e-4, mixed_precision=True,
                      output_types=["state", "mean", "max"], save_every=0.5, summarise_every=0.5,
                      sample_summaries_every=0.125, save_variables=[f"V{j:02d}" for j in range(nc)],
                      summarise_variables=[f"V{j:02d}" for j in range(nc)])
    if kind == "fhn_fit":
        return Solver(_system("fhn", False), algorithm="dormand-prince-54", rtol=1e-6, atol=1e-6,
                      output_types=["state"], saved_state_indices=[0], save_every=1.0, mixed_precision=True,
                      adjoint=True)
    if kind == "vdp_fit":
        return Solver(_system("vdp", False), algorithm="ros3p", linear_correction_type="direct",
                      preconditioner_type=None, rtol=1e-6, atol=1e-6, output_types=["state"],
                      saved_state_indices=[0], save_every=1.0, mixed_precision=True, adjoint=True)
    common = dict(rtol=1e-4, output_types=["state"], mixed_precision=True)
    direct = dict(linear_correction_type="direct", preconditioner_type=None)
    return HeteroSolver([
        Solver(_system("lorenz", False), algorithm="dormand-prince-54", atol=1e-8, **common),
        Solver(_system("vdp", False), algorithm="ros3p", atol=1e-8, save_variables=["x"], **direct, **common),
        Solver(_system("robertson", False), algorithm="ros3p", atol=1e-10, **direct, **common)])


class _State:
    pass


def prepare(case, seed):
    kind = case["kind"]
    data = _inputs(case, seed)
    ptype, _ = _precision(case)
    s = _State()
    s.case = case
    s.solver = _solver(kind, case.get("algorithm"), case.get("linear"), case.get("precision", "mixed"),
                       case.get("compartments", 0))
    if kind == "mixed":
        s.batches = [dict(initial_values=torch.tensor(f["x0"], dtype=torch.float32, device="cuda"),
                          parameters=torch.tensor(f["p"], dtype=torch.float32, device="cuda"),
                          duration=float(f["durations"].max()), durations=f["durations"],
                          tol_scale=f["tol_scale"]) for f in data["families"]]
        return s
    if kind in ("lorenz", "lorenz_rows") and case.get("host"):
        # arrays of the program, as the reference's users pass them
        s.x0, s.p = data["x0"].astype(ptype), data["p"].astype(ptype)
    elif case.get("host"):
        s.x0, s.p = (torch.tensor(data[k].astype(ptype)).pin_memory() for k in ("x0", "p"))
    else:
        s.x0, s.p = (torch.tensor(data[k].astype(ptype), device="cuda") for k in ("x0", "p"))
    if "durations" in data:
        d = torch.tensor(data["durations"])
        s.durations = d.pin_memory() if case.get("host") else d.cuda()
        s.longest = float(data["durations"].max())
    if "samples" in data:
        name, period = ("F", 0.25) if kind == "driven" else ("I", 0.1)
        s.drivers = ArrayInterpolator(np.float32, {name: data["samples"], "driver_sample_period": period, "t0": 0.0,
                                                   "wrap": True}, [name])
    if "target" in data:
        s.target = torch.tensor(data["target"], dtype=torch.float32, device="cuda")
        s.integrator = AdjointIntegrator(s.solver, ckpt_every=64, max_ckpts=64)
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "lorenz":
        r = s.solver.solve(s.x0, s.p, duration=case["horizon"], on_device=not case["host"])
        return r.state, r.status_codes
    if kind == "lorenz_rows":
        r = s.solver.solve(s.x0, s.p, duration=0.01 * (case["rows"] // 10 * 10), on_device=True)
        return r.state, r.state_summaries, r.status_codes
    if kind == "vdp":
        r = s.solver.solve(s.x0, s.p, duration=s.longest, durations=s.durations, on_device=not case["host"])
        return r.state, r.status_codes
    if kind == "driven":
        r = s.solver.solve(s.x0, s.p, drivers=s.drivers, duration=0.5 * case["rows"], on_device=True)
        return r.state, r.observables, r.status_codes
    if kind == "cable":
        r = s.solver.solve(s.x0, s.p, drivers=s.drivers, duration=case["horizon"], on_device=True)
        return r.state, r.state_summaries, r.status_codes
    if kind in ("fhn_fit", "vdp_fit"):
        # one step of a fit: squared distance of the saved rows to the targets
        state, status, saved = s.integrator.forward(s.x0, s.p, float(case["horizon"]))
        grad = (2.0 / state.shape[0]) * (state - s.target[:, None])
        grad_x0, grad_p = s.integrator.backward(saved, grad)
        return state, grad_x0, grad_p, status
    out = []
    for r in s.solver.solve(s.batches, on_device=True):
        out += [r.state, r.status_codes]
    return out


# Attempted steps of one run (mean over the inputs' distribution, measured)
# and the operations of one step, counted from the methods' formulas; they
# size ``work`` only.
def work(case):
    n, kind = case["runs"], case["kind"]
    size = 8 if case.get("precision") == "float64" else 4
    if kind == "lorenz":
        steps = case["horizon"] * (207 if size == 8 else 61)
        return {"bytes": n * (7 * size + 4 + 6 * size), "flops": n * steps * 210}
    if kind == "lorenz_rows":
        rows = case["rows"] // 10 * 10
        steps = rows * (2.1 if size == 8 else 1.1)
        return {"bytes": n * (4 * size + 3 * size * (rows + 1) + 6 * size * (rows // 10) + 4),
                "flops": n * steps * 210}
    if kind == "vdp":
        steps, per = (670, 190) if case["algorithm"] == "ros3p" else (560, 1500)
        steps = 1900 if case.get("spread") else steps
        return {"bytes": n * (3 * size + 8 + 2 * size + 4), "flops": n * steps * per}
    if kind == "driven":
        return {"bytes": n * (16 + 16 * (case["rows"] + 1) + 4), "flops": n * case["rows"] * 2900}
    if kind == "cable":
        nc, h = case["compartments"], case["horizon"]
        rows = int(round(2 * h))
        return {"bytes": n * (16 * nc + 12 + 4 * nc * (3 * rows + 1) + 4), "flops": n * h * nc * 59e3}
    if kind == "fhn_fit":
        rows = case["horizon"] + 1
        return {"bytes": n * (24 * 2 + 8 * rows + 4), "flops": n * case["horizon"] * 2.2 * 900}
    if kind == "vdp_fit":
        rows = case["horizon"] + 1
        return {"bytes": n * (12 * 2 + 8 * rows + 4), "flops": n * case["horizon"] * 14 * 700}
    return {"bytes": n * 60, "flops": n * 400 * 200}


# About four times the largest 2-norm error of any output against ``exact``,
# or (``spread``, which has no exact values) against the same path compiled
# without fast math, over several seeds at the listed sizes.  Adaptive solves
# carry their method's error at the tolerance they ask for, far above the
# rounding of their type; the runs that end inside a relaxation jump make up
# the error of the spread ensemble.
def tolerance(case):
    kind, double = case["kind"], case.get("precision") == "float64"
    if kind == "lorenz":
        return {"rel": 2e-7 if double else 7e-5}
    if kind == "lorenz_rows":
        return {"rel": 1e-8 if double else 5e-5}
    if kind == "vdp":
        return {"rel": 2e-2 if case.get("spread") else 2e-6}
    return {"rel": {"driven": 6e-4, "cable": 2e-6, "fhn_fit": 2e-5, "vdp_fit": 4e-5, "mixed": 1.2e-4}[kind]}


# ---------------------------------------------------------------------------
# FP64 values
# ---------------------------------------------------------------------------
def _gbs(f, y, t, h, steps, columns, row=None):
    """Extrapolated modified midpoint over ``steps`` steps of ``h``."""
    n = [2 * (j + 1) for j in range(columns)]
    for k in range(steps):
        prev = []
        f0 = f(t, y)
        for j in range(columns):
            hj = h / n[j]
            a, b = y, y + hj * f0
            for i in range(1, n[j]):
                a, b = b, a + 2.0 * hj * f(t + i * hj, b)
            cur = [b if j == 0 else b]
            # Gragg's smoothing is not needed with an even number of substeps
            for q in range(1, j + 1):
                cur.append(cur[q - 1] + (cur[q - 1] - prev[q - 1]) / ((n[j] / n[j - q]) ** 2 - 1.0))
            prev = cur
        y = prev[-1]
        t = t + h
        if row is not None:
            row(k + 1, t, y)
    return y


def _inverse(A):
    """Inverse of ``[d, d, runs]`` matrices, d = 2 or 3."""
    if A.shape[0] == 2:
        det = A[0, 0] * A[1, 1] - A[0, 1] * A[1, 0]
        return torch.stack([torch.stack([A[1, 1], -A[0, 1]]), torch.stack([-A[1, 0], A[0, 0]])]) / det
    c = [torch.linalg.cross(A[(i + 1) % 3], A[(i + 2) % 3], dim=0) for i in range(3)]
    det = (A[0] * c[0]).sum(0)
    return torch.stack(c, dim=1) / det


def _stiff(f, jac, y0, p0, horizon, rtol=1e-11, atol=1e-14, columns=8):
    """Extrapolated linearly implicit Euler with its own step size per run
    (autonomous systems)."""
    out = y0.clone()
    live = torch.arange(y0.shape[1], device=y0.device)
    y, p, T = y0, p0, horizon
    t, h = torch.zeros_like(T), 1e-3 * torch.clamp(T, max=1.0)
    eye = torch.eye(y0.shape[0], dtype=y0.dtype, device=y0.device)[:, :, None]
    for it in range(100000):
        last = h >= T - t
        hh = torch.where(last, T - t, h)
        J = jac(y, p)
        prev = None
        for j in range(columns):
            hj = hh / (j + 1)
            Ai = _inverse(eye - hj * J)
            z = y
            for _ in range(j + 1):
                z = z + (Ai * (hj * f(z, p))[None]).sum(1)
            cur = [z]
            for q in range(1, j + 1):
                cur.append(cur[q - 1] + (cur[q - 1] - prev[q - 1]) / ((j + 1) / (j + 1 - q) - 1.0))
            before, prev = (prev[-1] if prev else None), cur
        new = prev[-1]
        scale = atol + rtol * torch.maximum(y.abs(), new.abs())
        err = ((new - prev[-2]).abs() / scale).amax(0)
        err = torch.where(torch.isfinite(err), err, torch.full_like(err, 1e12))
        ok = err <= 1.0
        gain = torch.clamp(0.85 * torch.clamp(err, min=1e-10) ** (-1.0 / columns), 0.1, 3.0)
        y = torch.where(ok, new, y)
        t = torch.where(ok, torch.where(last, T, t + hh), t)
        h = hh * gain
        if it % 16 == 15:
            done = t >= T
            if bool(done.any()):
                out[:, live[done]] = y[:, done]
                keep = ~done
                live, y, p, T, t, h = live[keep], y[:, keep], p[:, keep], T[keep], t[keep], h[keep]
            if live.numel() == 0:
                return out
    return None


def _periodic_spline(samples, period):
    """Value function of the periodic cubic spline through ``samples``."""
    y = np.asarray(samples, dtype=np.float64)[:-1]
    m = y.size
    A = 4.0 * np.eye(m) + np.roll(np.eye(m), 1, axis=1) + np.roll(np.eye(m), -1, axis=1)
    M = np.linalg.solve(A, 6.0 * (np.roll(y, -1) - 2.0 * y + np.roll(y, 1)))  # second derivatives, unit spacing

    def value(t):
        u = t / period
        k = math.floor(u + 1e-12)
        x = u - k
        i, j = k % m, (k + 1) % m
        return float((1 - x) * y[i] + x * y[j] + ((1 - x) ** 3 - (1 - x)) * M[i] / 6.0 + (x ** 3 - x) * M[j] / 6.0)
    return value


def _dev(a, dtype=np.float64):
    """Inputs as the solver receives them (rounded to its precision), in FP64 on the GPU."""
    return torch.tensor(np.asarray(a, dtype=dtype).astype(np.float64), device="cuda" if torch.cuda.is_available() else "cpu")


def _f_lorenz(y, rho, scale=1.0):
    return torch.stack([SIGMA * (y[1] - y[0]), y[0] * (rho - y[2]) - y[1], y[0] * y[1] - BETA * y[2]]) * scale


def _f_vdp(y, p):
    return torch.stack([y[1], p[0] * (1.0 - y[0] ** 2) * y[1] - y[0]])


def _j_vdp(y, p):
    one = torch.ones_like(y[0])
    return torch.stack([torch.stack([0.0 * one, one]),
                        torch.stack([-2.0 * p[0] * y[0] * y[1] - 1.0, p[0] * (1.0 - y[0] ** 2)])])


def _f_rob(y, k):
    a, b, c = k[0] * y[0], k[2] * y[1] * y[2], k[1] * y[1] ** 2
    return torch.stack([b - a, a - b - c, c])


def _j_rob(y, k):
    z = torch.zeros_like(y[0])
    d2 = 2.0 * k[1] * y[1]
    r0 = torch.stack([-k[0], k[2] * y[2], k[2] * y[1]])
    return torch.stack([r0, torch.stack([k[0], -k[2] * y[2] - d2, -k[2] * y[1]]), torch.stack([z, d2, z])])


def _status(n):
    return torch.zeros(n, dtype=torch.int32)


def exact(case, seed):
    kind, n = case["kind"], case["runs"]
    data = _inputs(case, seed)
    ptype, _ = _precision(case)
    if kind == "mixed":
        x, k, d = (_dev(data["families"][0][q], np.float64 if q == "durations" else np.float32)
                   for q in ("x0", "p", "durations"))
        out = [torch.stack([x, _gbs(lambda t, y: _f_lorenz(y, k[0], d), x, 0.0, 1.0 / 200, 200, 6)]).cpu(),
               _status(n // 3)]
        for fam, f, j in ((1, _f_vdp, _j_vdp), (2, _f_rob, _j_rob)):
            x, k, d = (_dev(data["families"][fam][q], np.float64 if q == "durations" else np.float32)
                       for q in ("x0", "p", "durations"))
            end = _stiff(f, j, x, k, d, atol=1e-16 if fam == 2 else 1e-14)
            rows = torch.stack([x, end])
            out += [(rows[:, :1] if fam == 1 else rows).cpu(), _status(n // 3)]
        return out
    x0, p = _dev(data["x0"], ptype), _dev(data["p"], ptype)
    if kind == "lorenz":
        steps = 100
        y = _gbs(lambda t, y: _f_lorenz(y, p[0]), x0, 0.0, case["horizon"] / (2 * steps), 2 * steps, 6)
        return torch.stack([x0, y]).cpu(), _status(n)
    if kind == "lorenz_rows":
        rows = [x0]
        _gbs(lambda t, y: _f_lorenz(y, p[0]), x0, 0.0, 0.01, case["rows"] // 10 * 10, 6,
             lambda k, t, y: rows.append(y))
        rows = torch.stack(rows)
        w = rows[1:].reshape(-1, 10, 3, n)
        return rows.cpu(), torch.stack([w.mean(1), w.amax(1)], dim=2).reshape(w.shape[0], 6, n).cpu(), _status(n)
    if kind == "vdp":
        if n > 100000:
            return None
        end = _stiff(_f_vdp, _j_vdp, x0, p, _dev(data["durations"]))
        return torch.stack([x0, end])[:, :1].cpu(), _status(n)
    if kind == "driven":
        force = _periodic_spline(data["samples"], 0.25)
        rows, per = [x0], 10
        _gbs(lambda t, y: torch.stack([y[1], force(t) - p[0] * y[0] - p[1] * y[1]]), x0, 0.0, 0.5 / per,
             per * case["rows"], 4, lambda k, t, y: rows.append(y) if k % per == 0 else None)
        y = torch.stack(rows)
        times = (0.5 * torch.arange(y.shape[0], dtype=torch.float64, device=y.device))[:, None].expand(-1, n)
        return (torch.cat([y, times[:, None]], dim=1).cpu(),
                (0.5 * y[:, 1] ** 2 + 0.5 * p[0] * y[:, 0] ** 2)[:, None].cpu(), _status(n))
    if kind == "cable":
        return _exact_cable(case, data, x0, p)
    if n * case["horizon"] > 131072 * 60:
        return None
    return _exact_fit(case, data, x0, p)


def _exact_fit(case, data, x0, p):
    """States and loss gradients from the variational equations."""
    n, T = case["runs"], case["horizon"]
    np_ = p.shape[0]
    m = 2 + np_

    if case["kind"] == "fhn_fit":
        a, b, tau, cur = p
        zero, one = torch.zeros_like(a), torch.ones_like(a)

        def parts(v, w):
            f = (v - v ** 3 / 3.0 - w + cur, (v + a - b * w) / tau)
            J = (1.0 - v ** 2, -one, one / tau, -b / tau)
            P = ((zero, zero, zero, one), (one / tau, -w / tau, -f[1] / tau, zero))
            return f, J, P
    else:
        mu = p[0]

        def parts(x, y):
            s = (1.0 - x ** 2) * y
            f = (y, mu * s - x)
            J = (torch.zeros_like(x), torch.ones_like(x), -2.0 * mu * x * y - 1.0, mu * (1.0 - x ** 2))
            P = ((torch.zeros_like(x),), (s,))
            return f, J, P

    def rhs(t, z):
        f, J, P = parts(z[0], z[1])
        S = z[2:].reshape(2, m, n)
        d0 = J[0] * S[0] + J[1] * S[1]
        d1 = J[2] * S[0] + J[3] * S[1]
        for q in range(np_):
            d0[2 + q] += P[0][q]
            d1[2 + q] += P[1][q]
        return torch.cat([f[0][None], f[1][None], d0, d1])

    S0 = torch.zeros((2, m, n), dtype=x0.dtype, device=x0.device)
    S0[0, 0] = 1.0
    S0[1, 1] = 1.0
    z = torch.cat([x0, S0.reshape(2 * m, n)])
    target = _dev(data["target"], np.float32)
    rows = [x0[0]]
    weight = 2.0 / (T + 1)
    grad = weight * (x0[0] - target[0]) * S0[0]
    per = 4 if case["kind"] == "fhn_fit" else 20

    def row(k, t, y):
        nonlocal grad
        if k % per == 0:
            rows.append(y[0])
            grad = grad + weight * (y[0] - target[k // per]) * y[2:2 + m]

    _gbs(rhs, z, 0.0, 1.0 / per, per * T, 5, row)
    return torch.stack(rows)[:, None].cpu(), grad[:2].cpu(), grad[2:].cpu(), _status(n)


def _exact_cable(case, data, x0, p):
    """The three-stage L-stable DIRK with fixed steps, its stages solved to
    FP64 rounding: gates eliminated, a dense solve for the voltages."""
    n, nc = case["runs"], case["compartments"]
    if n * nc * nc > 7000000:
        return None
    steps = int(round(case["horizon"] * 32))
    arc = math.atan(math.sqrt(2.0) / 4.0) / 3.0
    g = 1.0 + (math.sqrt(6.0) * math.sin(arc) - math.sqrt(2.0) * math.cos(arc)) / 2.0
    b1, b2 = (-6.0 * g * g + 16.0 * g - 1.0) / 4.0, (6.0 * g * g - 20.0 * g + 5.0) / 4.0
    a = ((), ((1.0 - g) / 2.0,), (b1, b2))
    c = (g, (1.0 + g) / 2.0, 1.0)
    current = _periodic_spline(data["samples"], 0.1)
    gna, gk, gc = (q[:, None] for q in p)
    y = x0.reshape(4, nc, n).permute(0, 2, 1).contiguous()           # [4, run, compartment]
    lap = torch.zeros((nc, nc), dtype=y.dtype, device=y.device)
    for i in range(nc):
        for j in (i - 1, i + 1):
            if 0 <= j < nc:
                lap[i, j] += 1.0
                lap[i, i] -= 1.0
    h = 0.03125

    def rates(v):
        """alpha, beta and their derivatives of the gates m, h, n."""
        out = []
        for s, v0, w in ((0.1, 40.0, None), (None, None, None), (0.01, 55.0, None)):
            if s is None:
                e = torch.exp(-(v + 65.0) / 20.0)
                al, dal = 0.07 * e, -0.07 / 20.0 * e
                e = torch.exp(-(v + 35.0) / 10.0)
                be = 1.0 / (1.0 + e)
                dbe = be * be * e / 10.0
            else:
                e = torch.exp(-(v + v0) / 10.0)
                q = 1.0 - e
                al = s * (v + v0) / q
                dal = s / q - s * (v + v0) * e / (10.0 * q * q)
                k, w = (4.0, 18.0) if s == 0.1 else (0.125, 80.0)
                be = k * torch.exp(-(v + 65.0) / w)
                dbe = -be / w
            out.append((al, be, dal, dbe))
        return out

    def field(z, cur):
        v, m_, h_, n_ = z
        f = gc * (v @ lap) - gna * m_ ** 3 * h_ * (v - 50.0) - gk * n_ ** 4 * (v + 77.0) - 0.3 * (v + 54.4)
        f[:, 0] += cur
        return torch.stack([f] + [al * (1.0 - x) - be * x for (al, be, _, _), x in zip(rates(v), (m_, h_, n_))])

    def stage(base, cur, guess):
        z = guess
        for _ in range(12):
            v, m_, h_, n_ = z
            r = base + h * g * field(z, cur) - z
            # gate rows: dx (1 + h g (al + be)) - h g (dal (1 - x) - dbe x) dv = r
            dv_diag = -gna * m_ ** 3 * h_ - gk * n_ ** 4 - 0.3
            dg = (-3.0 * gna * m_ ** 2 * h_ * (v - 50.0), -gna * m_ ** 3 * (v - 50.0), -4.0 * gk * n_ ** 3 * (v + 77.0))
            diag, rhs, gates = 1.0 - h * g * dv_diag, r[0].clone(), []
            for (al, be, dal, dbe), x, d, rx in zip(rates(v), (m_, h_, n_), dg, r[1:]):
                den = 1.0 + h * g * (al + be)
                k = h * g * (dal * (1.0 - x) - dbe * x) / den
                gates.append((rx / den, k))
                rhs += h * g * d * rx / den
                diag = diag - h * g * d * k
            A = torch.diag_embed(diag) - (h * g * gc)[:, :, None] * lap
            dv = torch.linalg.solve(A, rhs)
            step = torch.stack([dv] + [c0 + k * dv for c0, k in gates])
            z = z + step
            if float((step.abs() / (1e-3 + z.abs())).max()) < 1e-12:
                break
        return z

    saved, means, maxs, acc = [y[0].T.clone()], [], [], []
    for k in range(steps):
        fs = []
        for i in range(3):
            base = y + h * sum(w * f for w, f in zip(a[i], fs)) if i else y
            cur = current((k + c[i]) * h)
            z = stage(base, cur, y if i == 0 else z)
            fs.append((z - base) / (h * g))
        y = y + h * (b1 * fs[0] + b2 * fs[1] + g * fs[2])
        if (k + 1) % 4 == 0:
            acc.append(y[0].T.clone())
        if (k + 1) % 16 == 0:
            saved.append(y[0].T.clone())
            w = torch.stack(acc)
            means.append(w.mean(0))
            maxs.append(w.amax(0))
            acc = []
    summ = torch.stack([torch.stack([m, x], dim=1).reshape(2 * nc, n) for m, x in zip(means, maxs)])
    return torch.stack(saved).cpu(), summ.cpu(), _status(n)
