"""Per-run horizons and tolerance scales reach the device with one entry per
run: the claim-order kernels and the integration read that many (CPU)."""

import numpy as np
import pytest
import torch


def test_claim_order_reads_one_entry_per_run():
    from cubie_b200.solver import Solver
    work = torch.tensor([3.0, 1.0, 2.0], dtype=torch.float64)
    assert Solver._claim_work(work) == (work, None)
    for scale in (torch.tensor([0.5, 1.0, 2.0]), torch.tensor([0.5], dtype=torch.float64), torch.tensor(0.5)):
        horizon, s = Solver._claim_work(work, scale)
        assert horizon is work
        assert s.dtype == torch.float64 and s.is_contiguous() and s.numel() == work.numel()
        np.testing.assert_array_equal(s.numpy(), np.broadcast_to(scale.numpy(), 3))
    # left to the general path: fewer or more scales than runs, another
    # device, other layouts and types of the horizons, no runs
    for scale in (torch.ones(2), torch.ones(4), torch.ones((3, 1)), torch.ones(3, device="meta")):
        assert Solver._claim_work(work, scale) is None
    for horizon in (work.float(), torch.ones((6,), dtype=torch.float64)[::2], work[None], work[:0]):
        assert Solver._claim_work(horizon, None) is None


def test_general_path_refuses_a_wrong_number_of_scales():
    from cubie_b200 import Solver, create_ODE_system
    sysm = create_ODE_system(["dx = -k * x"], states=["x"], parameters=["k"], precision=np.float32)
    s = Solver(sysm, algorithm="tsit5", output_types=["state"])
    with pytest.raises(RuntimeError):
        s.run_order(torch.ones(3, dtype=torch.float64), torch.ones(2, dtype=torch.float64))


def test_mixed_batch_inputs_have_one_entry_per_run():
    from cubie_b200.hetero import _per_run
    assert _per_run(None, 3, "durations", "cpu") is None
    for values in ([1.0, 2.0, 3.0], np.ones((1, 3), np.float32), torch.ones(3)):
        t = _per_run(values, 3, "durations", "cpu")
        assert t.dtype == torch.float64 and tuple(t.shape) == (3,)
    for values in ([1.0], np.ones(2), torch.ones(4), 2.0):
        with pytest.raises(ValueError, match="tol_scale must have one entry per run"):
            _per_run(values, 3, "tol_scale", "cpu")
