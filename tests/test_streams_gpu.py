"""Solves on a stream of the caller's: the inputs, cleared buffers and claim
orders are queued on torch's current stream, so the launch waits for it.  With
the current stream kept busy beforehand the results are the default stream's,
bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VDP = ["dx = y", "dy = mu * (1 - x**2) * y - x"]
LORENZ = ["dx = 10.0 * (y - x)", "dy = x * (rho - z) - y", "dz = x * y - 2.5 * z"]


def _keep_busy():
    """Some milliseconds of work on the current stream."""
    import torch
    a = torch.ones((4096, 4096), device="cuda")
    for _ in range(20):
        a = a @ a * 1e-4
    return a


def _vdp(**kw):
    from cubie_b200 import Solver, create_ODE_system
    sysm = create_ODE_system(VDP, states=["x", "y"], parameters=["mu"], precision=np.float32)
    return Solver(sysm, algorithm="ros3p", linear_correction_type="direct", preconditioner_type=None, rtol=1e-5,
                  atol=1e-5, output_types=["state"], mixed_precision=True, **kw)


def _batch(n, seed=0):
    rng = np.random.default_rng(seed)
    mu = 10.0 ** rng.uniform(0, 2, n)
    return dict(initial_values=rng.uniform(-2, 2, (2, n)), parameters=mu[None], duration=1.0,
                durations=mu * rng.uniform(0.2, 1.0, n), tol_scale=10.0 ** rng.uniform(-1, 1, n))


# below and above the one-block limit of the claim order
@pytest.mark.parametrize("n", [3000, 20011])
def test_solve_on_a_side_stream(cuda_device, n):
    import torch
    s, b = _vdp(), _batch(n)
    want = s.solve(**b)
    assert not want.status_codes.any()
    for _ in range(3):
        busy = _keep_busy()
        got = s.solve(**b, stream=torch.cuda.Stream())
        np.testing.assert_array_equal(got.state, want.state)
        np.testing.assert_array_equal(got.status_codes, want.status_codes)
        assert got.totals == want.totals
        del busy


def test_mixed_batch_on_a_side_stream(cuda_device):
    import torch
    from cubie_b200 import Solver, create_ODE_system
    from cubie_b200.hetero import HeteroSolver
    sysm = create_ODE_system(LORENZ, states=["x", "y", "z"], parameters=["rho"], precision=np.float32)
    lorenz = Solver(sysm, algorithm="tsit5", rtol=1e-5, atol=1e-5, output_types=["state"], mixed_precision=True)
    rng = np.random.default_rng(1)
    batches = [dict(initial_values=rng.uniform(-10, 10, (3, 5001)), parameters=rng.uniform(20, 30, (1, 5001)),
                    duration=1.0), _batch(5003)]
    h = HeteroSolver([lorenz, _vdp()], fp32_floor=None, mixed_floor=None)
    want = h.solve(batches)
    for _ in range(3):
        busy = _keep_busy()
        got = h.solve(batches, stream=torch.cuda.Stream())
        for g, w in zip(got, want):
            assert not w.status_codes.any()
            np.testing.assert_array_equal(g.state, w.state)
            assert g.totals == w.totals
        del busy


def test_chunks_wait_for_their_cleared_buffers(cuda_device):
    s, b = _vdp(), _batch(2000)
    want = s.solve(**b)
    chunked = _vdp(max_chunk_runs=640)
    busy = _keep_busy()
    got = chunked.solve(**b)
    assert chunked.chunks > 1
    np.testing.assert_array_equal(got.state, want.state)
    assert got.totals == want.totals
    del busy
