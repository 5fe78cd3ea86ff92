"""Claim order of a persistent launch on the device: a permutation of the
runs by decreasing estimated work, to within a bin's width (2^(1/16))."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver():
    from cubie_b200 import Solver, create_ODE_system
    sysm = create_ODE_system(["dx = y", "dy = mu * (1 - x**2) * y - x"], states=["x", "y"], parameters=["mu"],
                             precision=np.float32)
    return Solver(sysm, algorithm="ros3p", output_types=["state"])


# one block, its limit, the first size of the tiled launches, a ragged last
# tile, more tiles than one wave
@pytest.mark.parametrize("n", [1, 31, 1025, 4096, 4097, 40961, 700001])
@pytest.mark.parametrize("scaled", [False, True])
def test_order_is_a_sorted_permutation(cuda_device, n, scaled):
    import torch
    rng = np.random.default_rng(n)
    work = torch.tensor(10.0 ** rng.uniform(-3, 4, n), device="cuda")
    scale = torch.tensor(10.0 ** rng.uniform(-4, 0, n), device="cuda") if scaled else None
    order = _solver().run_order(work, scale)
    assert order.dtype == torch.int64
    assert torch.equal(torch.sort(order).values, torch.arange(n, device="cuda"))
    cost = work if scale is None else work * scale ** -0.25
    c = cost[order]
    # every claim costs at most a bin (and FP32 rounding) more than any before it
    assert bool((c <= 2.0 ** (1.001 / 16) * torch.cummin(c, 0).values).all())


@pytest.mark.parametrize("n", [1000, 50000])
def test_odd_horizons_keep_a_permutation(cuda_device, n):
    import torch
    work = torch.full((n,), 5.0, dtype=torch.float64, device="cuda")
    work[::7] = 0.0
    work[3::11] = float("nan")
    work[5::13] = -1.0
    work[6::17] = float("inf")
    work[8::19] = 1e300
    scale = torch.ones_like(work)
    scale[::5] = 0.0
    for s in (None, scale):
        order = _solver().run_order(work, s)
        assert torch.equal(torch.sort(order).values, torch.arange(n, device="cuda"))
