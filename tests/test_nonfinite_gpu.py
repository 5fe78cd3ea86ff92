"""Runs that start at NaN or infinity stop with an error status (or their
step budget) and leave the other runs of the batch untouched, bit for bit:
the norms, clamps and limits pass a NaN on instead of dropping it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VDP = ["dx = y", "dy = mu * (1 - x**2) * y - x"]


@pytest.mark.parametrize("algorithm,linear,kind", [
    ("dormand-prince-54", "minimal_residual", "mixed"), ("dormand-prince-54", "minimal_residual", "float32"),
    ("ros3p", "direct", "mixed"), ("ros3p", "minimal_residual", "float32"), ("radau", "gmres", "mixed"),
    ("l_stable_sdirk_4", "bicgstab", "float32"), ("kvaerno3", "direct", "float64")])
def test_nonfinite_runs_stay_alone(cuda_device, algorithm, linear, kind):
    from cubie_b200 import Solver, create_ODE_system
    p = np.float64 if kind == "float64" else np.float32
    sysm = create_ODE_system(VDP, states=["x", "y"], parameters=["mu"], precision=p)
    s = Solver(sysm, algorithm=algorithm, linear_correction_type=linear, mixed_precision=kind == "mixed",
               rtol=1e-4, atol=1e-4, output_types=["state"], max_steps=2000)
    rng = np.random.default_rng(1)
    x0, mu = rng.uniform(-2, 2, (2, 40)), rng.uniform(1, 5, (1, 40))
    good = s.solve(x0, mu, duration=2.0, nan_error_trajectories=False)
    assert not good.status_codes.any()
    bad = x0.copy()
    bad[0, 3], bad[1, 17], bad[0, 31] = np.nan, np.inf, -np.inf
    r = s.solve(bad, mu, duration=2.0, nan_error_trajectories=False)
    hit = np.isin(np.arange(40), [3, 17, 31])
    assert np.all(r.status_codes[hit] != 0)
    assert not r.status_codes[~hit].any()
    np.testing.assert_array_equal(r.state[:, :, ~hit], good.state[:, :, ~hit])
