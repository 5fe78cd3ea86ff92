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
    eqs += [f"dw{i:03d} = c * (u{i:03d} + 0.7 - 0.8 * w{i:03d})" for i in range(n)]
    names = [f"{v}{i:03d}" for i in range(n) for v in "uw"] if interleaved else \
        [f"{v}{i:03d}" for v in "uw" for i in range(n)]
    return eqs, {name: 0.1 for name in names}, {"k": 1.0, "c": 0.08}


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


def cable(nc):
    """The undriven Hodgkin-Huxley cable (tests/hh_models.py), grouped by variable."""
    from hh_models import hh_cable
    eqs, states, params, _ = hh_cable(nc)
    return [e.replace("I + ", "") for e in eqs], states, params


def scattered(n):
    """No constant offsets: every component reads another, in no pattern."""
    perm = np.random.default_rng(5).permutation(n)
    return ([f"du{i:03d} = k * u{perm[i]:03d} - 2 * u{i:03d} - c * u{i:03d}**3" for i in range(n)],
            {f"u{i:03d}": 0.1 for i in range(n)}, {"k": 1.0, "c": 0.08})


MODELS = {"cable19": cable(19), "interleaved33": ring(33, True), "ring21": ring(21), "scattered70": scattered(70),
          "ring128": ring(128)}
# expected form: (slots of the register form or 0, stride of its lanes)
FORMS = {"cable19": (4, 1), "interleaved33": (4, 2), "ring21": (2, 1), "scattered70": (0, 1), "ring128": (8, 1)}


def _model_inputs(name, n):
    if not name.startswith("cable"):
        return _inputs(len(MODELS[name][1]), n, 2)
    nc = int(name[5:])
    rng = np.random.default_rng(3)
    x0 = np.array(list(MODELS[name][1].values()))[:, None] \
        + rng.normal(0, 1, (4 * nc, n)) * np.repeat([8.0, 0.02, 0.02, 0.02], nc)[:, None]
    return x0, np.stack([rng.uniform(80, 160, n), rng.uniform(20, 50, n), rng.uniform(0.1, 1.0, n)])


def _units(a, b, tol):
    return float(np.max(np.abs(a - b) / (tol + tol * np.abs(b))))


# FP64: the ring of 128 exceeds the lanes' registers (832 bytes) and run in
# the shared-memory form although the generator offers the other one
@pytest.mark.parametrize("name,placement", [
    *((name, placement) for name in MODELS for placement in ("local", "shared", "registers") if name != "ring128"),
    ("ring128", "local")])
def test_forms_match_the_oracle(cuda_device, name, placement):
    from oracle import OracleSystem, integrate
    model, n, T, tol = MODELS[name], 5, 0.5, 1e-8
    x0, p = _model_inputs(name, n)
    some = [0, 1, 31, 32, 33, x0.shape[0] - 1]       # ends of slots, a saved and summarised subset
    s = _solver(model, np.float64, rtol=tol, atol=tol, step_controller="fixed", dt=0.02, scratch_placement=placement,
                output_types=["state", "time", "mean", "max"], save_every=0.1, summarise_every=0.5,
                sample_summaries_every=0.1, summarised_state_indices=some)
    r = s.solve(x0, p, duration=T, nan_error_trajectories=False)
    code = s._system_code["warp"]
    source = s.prepare(T, load=False)["gen"].source
    assert (code.register_slots, 2 if "LANE_STRIDE = 2" in source else 1) == FORMS[name]
    eqs, states, params = model
    out = integrate(OracleSystem(eqs, list(states), list(params), {}), "l_stable_dirk_3", x0, p, T,
                    precision=np.float64, linear_correction_type="bicgstab", step_controller="fixed", dt=0.02,
                    save_every=0.1, dense_prediction=False, rtol=tol, atol=tol)
    assert r.status_codes.tolist() == [0] * n and out["status"].tolist() == [0] * n
    ns = x0.shape[0]
    # Newton stops below a tenth of the tolerance a stage; 25 steps of three
    # stages on flows that contract or grow by less than e
    assert _units(r.state[:, :ns], out["state"][:, :ns], tol) < 1.0
    rows = r.state[1:, some]                          # the samples of the one summary window
    np.testing.assert_allclose(r.state_summaries[0, 0::2], rows.mean(axis=0), rtol=1e-12, atol=1e-14)
    np.testing.assert_array_equal(r.state_summaries[0, 1::2], rows.max(axis=0))
