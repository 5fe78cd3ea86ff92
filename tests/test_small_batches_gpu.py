"""Persistent launches of batches smaller than the resident grid: the runs
are spread over one warp per scheduler, a few lanes of each; every run's
result is the plain one-thread-per-run launch's, bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one run, a block's worth and its neighbours, one run per warp (592 warps on
# 148 SMs) and its neighbours, a full warp per scheduler and its neighbours
@pytest.mark.parametrize("n", [1, 31, 128, 129, 591, 592, 593, 2500, 18943, 18944, 18945])
@pytest.mark.parametrize("block", [32, 128, 256])
def test_spread_batches_equal_plain_launches(cuda_device, n, block):
    from cubie_b200 import Solver, create_ODE_system
    sysm = create_ODE_system(["dx = y", "dy = mu * (1 - x**2) * y - x"], states=["x", "y"], parameters=["mu"],
                             precision=np.float32)
    rng = np.random.default_rng(n)
    x0, mu = rng.uniform(-2, 2, (2, n)), rng.uniform(1, 5, (1, n))
    out = []
    for kernel in ("persistent", "plain"):
        s = Solver(sysm, algorithm="dormand-prince-54", rtol=1e-4, atol=1e-4, output_types=["state"],
                   save_every=0.5, kernel=kernel, block_size=block)
        out.append(s.solve(x0, mu, duration=1.0))
    a, b = out
    assert not a.status_codes.any() and not b.status_codes.any()
    np.testing.assert_array_equal(a.state, b.state)
    assert a.totals == b.totals
