"""The FP64 controllers' powers on the device against extended precision:
no further from it than CUDA's pow, whose place they take.

Largest and root mean square error in units of the last place over 2^20 to
2^21 samples, norms from 1e-12 to 1e6: one power 1.07 and 0.31 (pow 1.32 and
0.39), two powers with their factor 1.52 and 0.44 (pow 3.59 and 0.72).  Norms
within 1e-3 to 10 under a small exponent are the narrowest case: 1.08 and 0.306
against 1.01 and 0.305, hence the allowances below (0.1 units and 2 %)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "cbx_common.cuh"
#include "cbx_args.h"
extern "C" __global__ void cbx_integrate_plain(cbx_solve_args args) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= args.n_runs) return;
    const double* in = static_cast<const double*>(args.inits);
    const double a = in[i], b = in[i + args.run_stride];
    static_cast<double*>(args.state_out)[i] = EXPRESSION;
}
"""


def _evaluate(expression, a, b):
    import torch
    from cubie_b200 import _native
    cubin, log = _native.compile_cubin(SOURCE.replace("EXPRESSION", expression), _native.default_options())
    mod = _native.Module(cubin, 0, log)
    x = torch.tensor(np.stack([a, b]), device="cuda")
    out, status = torch.empty_like(x[0]), torch.zeros(a.size, dtype=torch.int32, device="cuda")
    args = _native.SolveArgs()
    args.inits, args.state_out, args.status_out = x.data_ptr(), out.data_ptr(), status.data_ptr()
    args.n_runs = args.run_stride = a.size
    mod.launch(args, 0, 128, 0, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _ulps(got, want):
    return (np.abs(got.astype(np.longdouble) - want)
            / np.spacing(np.abs(want.astype(np.float64)))).astype(np.float64)


# norms of ordinary steps, of any step, and far beyond
RANGES = [(-3, 1), (-12, 6), (-60, 60), (-290, 290)]


@pytest.mark.parametrize("lo,hi", RANGES)
@pytest.mark.parametrize("order,kp", [(2, 0.7), (3, 1.0), (5, 0.7), (8, 0.25)])
def test_one_power(cuda_device, lo, hi, order, kp):
    a = 10.0 ** np.random.default_rng(order).uniform(lo, hi, 1 << 18)
    b = -kp / (2 * (order + 1))
    want = np.power(a.astype(np.longdouble), np.longdouble(b))
    ours, theirs = (_ulps(_evaluate(f"{f}(a, {b!r})", a, a), want) for f in ("cbx::pow_t", "pow"))
    assert ours.max() <= theirs.max() + 0.1
    assert np.sqrt(np.mean(ours ** 2)) <= 1.02 * np.sqrt(np.mean(theirs ** 2))


@pytest.mark.parametrize("lo,hi", RANGES[:3])
@pytest.mark.parametrize("order,kp,ki", [(3, 0.7, -0.4), (3, 1.0, 0.4), (5, 0.7, -0.4), (5, 0.7, 0.0), (8, 0.3, 0.2)])
def test_two_powers(cuda_device, lo, hi, order, kp, ki):
    rng = np.random.default_rng(order)
    a, b = 10.0 ** rng.uniform(lo, hi, 1 << 18), 10.0 ** rng.uniform(lo, 0, 1 << 18)
    x, y = -kp / (2 * (order + 1)), -ki / (2 * (order + 1))
    want = np.longdouble(0.9) * np.power(a.astype(np.longdouble), np.longdouble(x)) \
        * np.power(b.astype(np.longdouble), np.longdouble(y))
    ours = _ulps(_evaluate(f"cbx::scaled_powers(0.9, a, {x!r}, b, {y!r})", a, b), want)
    theirs = _ulps(_evaluate(f"0.9 * pow(a, {x!r}) * pow(b, {y!r})", a, b), want)
    assert ours.max() <= theirs.max() + 0.1
    assert np.sqrt(np.mean(ours ** 2)) <= 1.02 * np.sqrt(np.mean(theirs ** 2))


def test_ends_of_the_range_reach_the_clamp(cuda_device):
    """Zero, subnormal and infinite norms: a gain beyond any clamp, on pow's side."""
    a = np.array([0.0, 5e-324, 1e-310, 1.7e308, np.inf])
    for x, y in ((-0.0875, 0.05), (-0.125, -0.05), (-0.0389, 0.0222)):
        for got in (_evaluate(f"cbx::pow_t(a, {x!r})", a, a),
                    _evaluate(f"cbx::scaled_powers(0.9, a, {x!r}, b, {y!r})", a, np.ones_like(a))):
            assert np.all(got[:3] > 1e6) and np.all(got[3:] < 1e-6)
