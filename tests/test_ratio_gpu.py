"""The norms' FP64 quotient e / tol on the device against the division, over
the range of error terms and tolerances the norms meet."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "cbx_common.cuh"
#include "cbx_args.h"
extern "C" __global__ void cbx_integrate_plain(cbx_solve_args a) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n_runs) return;
    static_cast<double*>(a.state_out)[i] =
        cbx::ratio_t(static_cast<const double*>(a.inits)[i], static_cast<const double*>(a.params)[i]);
}
"""


def _ratios(e, tol):
    import torch
    from cubie_b200 import _native
    cubin, log = _native.compile_cubin(SOURCE, _native.default_options())
    mod = _native.Module(cubin, 0, log)
    x, t = torch.tensor(e, device="cuda"), torch.tensor(tol, device="cuda")
    out, status = torch.empty_like(x), torch.zeros(x.numel(), dtype=torch.int32, device="cuda")
    a = _native.SolveArgs()
    a.inits, a.params, a.state_out, a.status_out = (v.data_ptr() for v in (x, t, out, status))
    a.n_runs = a.run_stride = x.numel()
    mod.launch(a, 0, 128, 0, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def test_quotients_within_one_ulp(cuda_device):
    rng = np.random.default_rng(0)
    n = 1 << 20
    e = 10.0 ** rng.uniform(-30, 16, n) * rng.choice([-1.0, 1.0], n)
    tol = 10.0 ** rng.uniform(-16, 12, n)
    got, want = _ratios(e, tol), e / tol
    ulps = np.abs(got - want) / np.spacing(np.abs(want))
    assert float(ulps.max()) <= 1.0
    assert float(np.mean(ulps > 0)) < 1e-2          # nearly all are the division's own bits


def test_special_error_terms(cuda_device):
    e = np.array([0.0, np.inf, -np.inf, np.nan, 1e300, 1e16])
    tol = np.array([1e-6, 1e-6, 1e-6, 1e-6, 1e-12, 1e-16])
    with np.errstate(over="ignore"):
        np.testing.assert_array_equal(_ratios(e, tol), e / tol)


def test_quotients_have_the_divisions_bits(cuda_device):
    rng = np.random.default_rng(0)
    n = 1 << 20
    sign = rng.choice([-1.0, 1.0], n)
    ends = rng.integers(1, 64, n) * 2.0 ** -52       # mantissas at either end, where a reciprocal rounds worst
    for e, tol in ((10.0 ** rng.uniform(-30, 16, n) * sign, 10.0 ** rng.uniform(-16, 12, n)),
                   (np.ldexp(rng.uniform(1, 2, n), rng.integers(-500, 500, n)) * sign,
                    np.ldexp(rng.uniform(1, 2, n), rng.integers(-500, 500, n))),
                   (rng.uniform(1, 2, n), 2.0 - ends), (2.0 - ends, 1.0 + ends)):
        np.testing.assert_array_equal(_ratios(e, tol), e / tol)


def test_special_values_divide(cuda_device):
    """Zero, infinite and extreme tolerances, infinite and NaN terms."""
    terms = [0.0, 1e-200, 1e-16, 1.0, 1e16, 1e160, 1.7e308, np.inf]
    e, tol = (v.ravel().copy() for v in np.meshgrid([*terms, *(-v for v in terms), np.nan],
                                                    [0.0, 2.3e-308, 1e-200, 1e-16, 1.0, 1e160, 1e300, np.inf, np.nan]))
    with np.errstate(all="ignore"):
        want = e / tol
    keep = ~((np.abs(want) > 0) & (np.abs(want) < 1e-290))     # no quotient near the subnormal numbers
    np.testing.assert_array_equal(_ratios(e, tol)[keep], want[keep])


def test_infinite_constant_component_keeps_its_run(cuda_device):
    """A component that is infinite and stays so has an infinite tolerance:
    its ratio is zero and the others decide the step, in FP64 as in FP32."""
    from cubie_b200 import Solver, create_ODE_system
    for p in (np.float32, np.float64):
        sysm = create_ODE_system(["dx = -k * x", "dw = 0 * x"], states=["x", "w"], parameters=["k"], precision=p)
        s = Solver(sysm, algorithm="tsit5", rtol=1e-5, atol=1e-5, output_types=["state"])
        r = s.solve(np.array([[1.0, 1.0], [0.0, np.inf]]), np.ones((1, 2)), duration=1.0)
        assert r.status_codes.tolist() == [0, 0]
        assert abs(float(r.state[-1, 0, 1]) - np.exp(-1.0)) < 1e-4
