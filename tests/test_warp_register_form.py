"""Register form of the warp-per-system layout (CPU): the generated per-lane
functions, fed by the plan's exchanges carried out over 32 emulated lanes,
equal the straight-line right-hand side and Jacobian-vector product."""

import ctypes
import subprocess

import numpy as np
import pytest

from hh_models import hh_cable


def _ring(n):
    """A ring of n identical cells: every end couples across the whole vector."""
    eqs = [f"du{i:03d} = k * (u{(i - 1) % n:03d} - 2 * u{i:03d} + u{(i + 1) % n:03d}) - u{i:03d}**3 + w{i:03d}"
           for i in range(n)]
    eqs += [f"dw{i:03d} = 0.1 * (u{i:03d} - w{i:03d})" for i in range(n)]
    states = {**{f"u{i:03d}": 0.1 for i in range(n)}, **{f"w{i:03d}": 0.0 for i in range(n)}}
    return eqs, states, {"k": 1.0}, []


def _interleaved(n):
    """The ring with its cells' variables side by side."""
    eqs, states, params, drivers = _ring(n)
    order = [f"{v}{i:03d}" for i in range(n) for v in "uw"]
    return eqs, {k: states[k] for k in order}, params, drivers


def _scattered(n):
    """No constant offsets: every component reads another, in no pattern."""
    rng = np.random.default_rng(5)
    perm = rng.permutation(n)
    return ([f"du{i:03d} = k * u{perm[i]:03d} - u{i:03d}" for i in range(n)],
            {f"u{i:03d}": 0.1 for i in range(n)}, {"k": 1.0}, [])


def _code(model):
    from cubie_b200 import create_ODE_system
    from cubie_b200.codegen import generate_system
    from cubie_b200.warpgen import generate_warp_system
    eqs, states, params, drivers = model
    sysm = create_ODE_system(eqs, states=states, parameters=params, drivers=drivers, precision=np.float64)
    return sysm, generate_system(sysm), generate_warp_system(sysm)


# one slot, a slot shared by several variables, an odd size (a slot per
# variable), more than two slots; a multiple of 32 and not; ends that wrap over
# the whole vector; variables interleaved cell by cell
@pytest.mark.parametrize("model", [hh_cable(3), hh_cable(16), hh_cable(19), hh_cable(40), _ring(5), _ring(33),
                                   _interleaved(33), _interleaved(64)],
                         ids=["cable3", "cable16", "cable19", "cable40", "ring5", "ring33", "interleaved33",
                              "interleaved64"])
def test_lanes_equal_straight_line_code(model, tmp_path):
    sysm, g, w = _code(model)
    assert "NC = 0" not in w.source
    n = sysm.num_states
    src = ("#include <cmath>\n#define __device__\n#define __forceinline__ inline\n"
           "#define CBX_NOINLINE __attribute__((noinline))\nusing std::exp; using std::pow;\n"
           + g.source + "\n" + w.source + f"\nconstexpr int L = WarpSystem::SLOTS;\n" + r'''
using W = WarpSystem;
static void gather(const double loc[32][L], double g[32][W::NG > 0 ? W::NG : 1]) {
    for (int lane = 0; lane < 32; ++lane)
        for (int i = 0; i < W::NG; ++i) {
            const int from = (lane + W::g_shift(i)) & 31;            // the shuffle's source lane
            const bool first = W::g_mode(i) == 1 || (W::g_mode(i) == 0 && from >= W::g_shift(i));
            const int k = W::g_slot(i) + (first ? 0 : 1);
            g[lane][i] = (k >= 0 && k < L) ? loc[from][k] : 0.0;
        }
}
static void spread(const double* a, double loc[32][L]) {
    for (int lane = 0; lane < 32; ++lane)
        for (int k = 0; k < L; ++k)
            loc[lane][k] = lane < W::slot_count(k) ? a[W::slot_base(k) + lane * W::LANE_STRIDE] : 0.0;
}
extern "C" double eval(const double* y, const double* v, const double* p, const double* d, double* f1, double* j1,
                       double* f2, double* f3, double* j3) {
    System::dxdt<double>(y, p, d, 0.0, f1);
    double J[System::NJ]; System::jac<double>(y, p, d, 0.0, J); System::jmv<double>(J, v, j1);
    static double yl[32][L], vl[32][L], gy[32][W::NG > 0 ? W::NG : 1], gv[32][W::NG > 0 ? W::NG : 1];
    spread(y, yl); spread(v, vl); gather(yl, gy); gather(vl, gv);
    double padding = 0.0;
    for (int lane = 0; lane < 32; ++lane) {
        double fa[L], fb[L], jc[W::NC], jv[L];
        W::f_reg<double>(yl[lane], gy[lane], p, d, 0.0, lane, fa);
        W::fj_reg<double>(yl[lane], gy[lane], p, d, 0.0, lane, fb, jc);
        W::jmv_reg<double>(vl[lane], gv[lane], jc, jv);
        for (int k = 0; k < L; ++k) {
            const int c = W::slot_base(k) + lane * W::LANE_STRIDE;
            if (lane < W::slot_count(k)) { f2[c] = fa[k]; f3[c] = fb[k]; j3[c] = jv[k]; }
            else padding += std::fabs(fa[k]) + std::fabs(fb[k]) + std::fabs(jv[k]);
        }
    }
    return padding;
}
''')
    cpp, so = tmp_path / "wr.cpp", tmp_path / "wr.so"
    cpp.write_text(src)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", str(so), str(cpp)], check=True,
                   capture_output=True)
    lib = ctypes.CDLL(str(so))
    lib.eval.restype = ctypes.c_double
    lib.eval.argtypes = [ctypes.c_void_p] * 9
    rng = np.random.default_rng(0)
    y = rng.uniform(0.0, 1.0, n)
    if sysm.num_drivers:
        y[: n // 4] = rng.uniform(-80, 30, n // 4)
    v = rng.normal(size=n)
    p = np.array([120.0, 36.0, 0.5])
    d = np.array([3.0])
    f1, j1, f2, f3, j3 = (np.full(n, np.nan) for _ in range(5))   # every component is written
    padding = lib.eval(*[a.ctypes.data for a in (y, v, p, d, f1, j1, f2, f3, j3)])
    # the same expressions in another order of sums: a few roundings
    np.testing.assert_allclose(f2, f1, rtol=1e-13, atol=1e-12)
    np.testing.assert_allclose(f3, f1, rtol=1e-13, atol=1e-12)
    np.testing.assert_allclose(j3, j1, rtol=1e-12, atol=1e-10)
    assert padding == 0.0


def test_scattered_reads_keep_the_shared_form():
    _, _, w = _code(_scattered(64))
    assert "NC = 0, NG = 0" in w.source
