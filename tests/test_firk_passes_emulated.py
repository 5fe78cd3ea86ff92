"""Fully implicit steps taken one Newton iteration per pass (persistent
launch) against whole attempts (plain launch), device code emulated on the
CPU: the same bits, statuses and counts, through rejected attempts, Newton
failures, events, drivers and the end of the run."""

import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent / "host_emu"))

VDP = ["dx = y", "dy = mu * (1 - x**2) * y - x"]
DRIVEN = ["dx = v", "dv = -k * x - c * v + F"]


def _same(a, b):
    for key in ("state", "counters", "status", "totals", "state_sum"):
        if a[key] is not None:
            np.testing.assert_array_equal(a[key], b[key])


@pytest.mark.parametrize("algorithm", ["radau", "firk_gauss_legendre_2"])
@pytest.mark.parametrize("linear,kind,extra", [
    ("gmres", "mixed", {}), ("direct", "float32", {}), ("bicgstab", "float64", {}),
    ("gmres", "mixed", dict(newton_max_iters=1)),                          # steps that give up and are rejected
    ("direct", "mixed", dict(save_every=0.25, summarise_every=0.5, sample_summaries_every=0.25))])
def test_passes_equal_attempts(algorithm, linear, kind, extra):
    from emu import run_emulated
    from cubie_b200 import Solver, create_ODE_system
    p = np.float64 if kind == "float64" else np.float32
    sysm = create_ODE_system(VDP, states=["x", "y"], parameters=["mu"], precision=p)
    types = ["state", "iteration_counters"] + (["mean", "max"] if "summarise_every" in extra else [])
    s = Solver(sysm, algorithm=algorithm, linear_correction_type=linear, mixed_precision=kind == "mixed", rtol=1e-4,
               atol=1e-4, output_types=types, max_steps=3000, **extra)
    rng = np.random.default_rng(7)
    x0, mu = rng.uniform(-2, 2, (2, 9)), rng.uniform(1, 60, (1, 9))
    _same(run_emulated(s, x0, mu, 1.5, kernel="persistent"), run_emulated(s, x0, mu, 1.5, kernel="plain"))


def test_driven_passes_equal_attempts():
    from emu import run_emulated
    from cubie_b200 import Solver, create_ODE_system
    sysm = create_ODE_system(DRIVEN, states=["x", "v"], parameters=["k", "c"], drivers=["F"], precision=np.float64)
    s = Solver(sysm, algorithm="radau", rtol=1e-6, atol=1e-6, output_types=["state", "iteration_counters"],
               save_every=0.5)
    t = np.arange(41)
    drv = {"driver_sample_period": 0.25, "t0": 0.0, "wrap": True, "F": np.sin(2 * np.pi * t / 40) + (t == 40) * 0.0}
    drv["F"][-1] = drv["F"][0]
    rng = np.random.default_rng(8)
    x0, p = rng.uniform(-1, 1, (2, 5)), np.stack([rng.uniform(0.5, 4, 5), rng.uniform(0.1, 0.5, 5)])
    _same(run_emulated(s, x0, p, 3.0, kernel="persistent", drivers=drv),
          run_emulated(s, x0, p, 3.0, kernel="plain", drivers=drv))
