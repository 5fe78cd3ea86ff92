"""A solver's prepared launches (kernel source, module, output sizes) are used
again only under the settings they were prepared with (CPU)."""

import numpy as np
import pytest

DRIVEN = ["dx = v", "dv = -k * x - c * v + F"]


def _solver():
    from cubie_b200 import Solver, create_ODE_system
    sysm = create_ODE_system(DRIVEN, states=["x", "v"], parameters=["k", "c"], drivers=["F"], precision=np.float64)
    return Solver(sysm, algorithm="dormand-prince-54", rtol=1e-6, atol=1e-6, save_every=0.5,
                  output_types=["state", "time"])


def _interp(solver):
    from cubie_b200.interpolator import ArrayInterpolator
    samples = np.sin(2 * np.pi * np.arange(41) / 40)
    samples[-1] = samples[0]
    return ArrayInterpolator.from_system(
        solver.system, {"driver_sample_period": 0.25, "t0": 0.0, "wrap": True, "F": samples}, solver.precision)


def _assign(name, value):
    return lambda s: setattr(s, name, value)


@pytest.mark.parametrize("driven", [True, False])
@pytest.mark.parametrize("change,source", [
    (lambda s: s.rtol.__setitem__(slice(None), 1e-3), True), (_assign("dt_max", 0.125), True),
    (_assign("max_gain", 5.0), True), (_assign("saved_state_indices", [1]), True),
    (lambda s: s._user_timing.update(save_every=0.25), False), (_assign("block_size", 64), True),
    (lambda s: s.flags.update(time=False), True)])
def test_changed_settings_are_prepared_anew(driven, change, source):
    s = _solver()
    interp = _interp(s) if driven else None
    before = s.prepare(2.0, interp=interp, load=False)
    assert s.prepare(2.0, interp=interp, load=False) is before
    change(s)
    after = s.prepare(2.0, interp=interp, load=False)
    assert after is not before
    if source:
        assert after["gen"].key != before["gen"].key
    else:
        assert after["n_save"] != before["n_save"]
    assert s.prepare(2.0, interp=interp, load=False) is after


def test_threads_prepare_at_the_limit(monkeypatch):
    """Several threads at a full table: the oldest entries go, nothing raises."""
    import sys
    import threading
    from cubie_b200 import solver as solver_module
    s = _solver()
    interp = _interp(s)
    one = s.prepare(1.0, interp=interp, load=False)
    monkeypatch.setattr(solver_module, "PREPARED_MAX", 4)
    # the preparation itself takes milliseconds: without it the threads meet
    # at the table
    monkeypatch.setattr(s, "_generate", lambda spec: one["gen"])
    monkeypatch.setattr(s, "kernel_spec", lambda timing, meta=None: one["spec"])
    errors = []
    start = threading.Barrier(6)

    def work(k):
        start.wait()
        try:
            for i in range(400):
                s.prepare(1.0 + k + 1e-3 * i, interp=interp, load=False)
        except Exception as exc:
            errors.append(exc)

    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    try:
        threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    assert not errors
    assert len(s._prepared) <= 4 + 6
    s.prepare(99.0, interp=interp, load=False)
    assert len(s._prepared) <= 4
