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
