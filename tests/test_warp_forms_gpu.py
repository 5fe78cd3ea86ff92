"""The warp layout's two forms on the GPU (vectors in registers, or exchanged
through shared memory), over the lane maps of the register form: slots that
are only partly filled, variables interleaved cell by cell, couplings around
the whole vector."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ring(n, interleaved=False):
    """A ring of n FitzHugh-Nagumo cells."""
    eqs = [f"du{i:03d} = k * (u{(i - 1) % n:03d} - 2 * u{i:03d} + u{(i + 1) % n:03d}) + u{i:03d} - u{i:03d}**3 / 3"
           f" - w{i:03d} + 0.5" for i in range(n)]
    eqs += [f"dw{i:03d} = e * (u{i:03d} + 0.7 - 0.8 * w{i:03d})" for i in range(n)]
    names = [f"{v}{i:03d}" for i in range(n) for v in "uw"] if interleaved else \
        [f"{v}{i:03d}" for v in "uw" for i in range(n)]
    return eqs, {name: 0.1 for name in names}, {"k": 1.0, "e": 0.08}


def _inputs(n_states, n, seed=0):
    rng = np.random.default_rng(seed)
    return rng.normal(0, 1, (n_states, n)), np.stack([rng.uniform(0.2, 2, n), rng.uniform(0.05, 0.2, n)])


def _solver(model, precision, **kw):
    from cubie_b200 import Solver, create_ODE_system
    eqs, states, params = model
    sysm = create_ODE_system(eqs, states=states, parameters=params, precision=precision)
    base = dict(algorithm="l_stable_dirk_3", linear_correction_type="bicgstab", layout="warp",
                attempt_dense_prediction=False, output_types=["state"], rtol=1e-5, atol=1e-5)
    return Solver(sysm, **dict(base, **kw))


def test_runs_that_follow_one_another_in_a_warp(cuda_device):
    """More runs than resident warps, each with its own parameters: every run
    is what it is in a batch where it has a warp to itself, bit for bit."""
    s = _solver(ring(20), np.float32, step_controller="fixed", dt=0.05)
    x0, p = _inputs(40, 9000)
    whole = s.solve(x0, p, duration=0.5)
    assert not whole.status_codes.any()
    for first in (0, 4000, 8500):
        part = s.solve(x0[:, first:first + 500], p[:, first:first + 500], duration=0.5)
        np.testing.assert_array_equal(part.state, whole.state[:, :, first:first + 500])
