"""Launch bounds of the generated kernels: the generator's rule where the
caller named nothing, the caller's choice otherwise (CPU)."""

import re

import numpy as np
import pytest

from hh_models import hh_cable

VDP = ["dx = y", "dy = mu * (1 - x**2) * y - x"]


def _minimum(solver, macro="CBX_LAUNCH_BOUNDS"):
    """The minimum of blocks in the source's launch bounds; None: none asked."""
    m = re.search(rf"#define {macro}\(CFG\) __launch_bounds__\(CFG::BLOCK, (\d+)\)",
                  solver.prepare(2.0, load=False)["gen"].source)
    return None if m is None else int(m.group(1))


def _vdp(**kw):
    from cubie_b200 import Solver, create_ODE_system
    sysm = create_ODE_system(VDP, states=["x", "y"], parameters=["mu"], precision=np.float32)
    return Solver(sysm, output_types=["state"], **kw)


@pytest.mark.parametrize("algorithm,linear,rule", [("radau", "gmres", 2), ("radau", "direct", 2),
                                                   ("ros3p", "direct", 2), ("ros3p", "gmres", None),
                                                   ("tsit5", "minimal_residual", None),
                                                   ("l_stable_sdirk_4", "direct", None)])
def test_callers_choice_goes_before_the_rule(algorithm, linear, rule):
    kw = dict(algorithm=algorithm, linear_correction_type=linear)
    assert _minimum(_vdp(**kw)) == rule
    assert _minimum(_vdp(block_size=64, **kw)) == (None if rule is None else 4)
    assert _minimum(_vdp(block_size=512, **kw)) == (None if rule is None else 1)
    assert _minimum(_vdp(min_blocks_per_sm=1, **kw)) is None       # none asked for: none
    assert _minimum(_vdp(min_blocks_per_sm=5, **kw)) == 5
    assert _minimum(_vdp(max_registers=64, **kw)) is None          # a cap of the caller's own
    assert _minimum(_vdp(max_registers=64, min_blocks_per_sm=3, **kw)) == 3


@pytest.mark.parametrize("algorithm,linear", [("ros3p", "direct"), ("radau", "direct"), ("radau", "gmres")])
@pytest.mark.parametrize("n", [3, 4, 5, 8])
def test_rule_by_states(algorithm, linear, n):
    """Direct Rosenbrock steps are bounded up to four states, fully implicit
    ones always."""
    from cubie_b200 import Solver, create_ODE_system
    from cubie_b200.autotune import RULE_CANDIDATES, default_candidates
    if linear == "direct" and algorithm == "radau" and n > 4:
        linear = "gmres"                     # the operator of a direct solve is too wide
    sysm = create_ODE_system([f"du{i} = u{(i + 1) % n} - k * u{i}**3" for i in range(n)],
                             states=[f"u{i}" for i in range(n)], parameters=["k"], precision=np.float32)
    s = Solver(sysm, algorithm=algorithm, linear_correction_type=linear, output_types=["state"])
    bounded = algorithm == "radau" or n <= 4
    assert _minimum(s) == (2 if bounded else None)
    assert (RULE_CANDIDATES[0] in default_candidates(s)) == bounded


def test_warp_layout_takes_the_callers_choice():
    from cubie_b200 import Solver, create_ODE_system
    eqs, states, params, _ = hh_cable(64)
    sysm = create_ODE_system([e.replace("I + ", "") for e in eqs], states=states, parameters=params,
                             precision=np.float32)

    def minimum(**kw):
        return _minimum(Solver(sysm, algorithm="l_stable_dirk_3", linear_correction_type="bicgstab", layout="warp",
                               output_types=["state"], **kw), "CBX_WARP_BOUNDS")

    assert minimum() == 3                      # 12 warps at 128 threads
    assert minimum(min_blocks_per_sm=1) is None
    assert minimum(min_blocks_per_sm=2) == 2
    assert minimum(max_registers=168) is None


def test_autotuner_tries_the_rule_and_none():
    from cubie_b200.autotune import DEFAULT_CANDIDATES, default_candidates
    bounded = default_candidates(_vdp(algorithm="radau", linear_correction_type="gmres"))
    assert {(128, 0), (128, 1), (64, 0), (64, 1)} <= set(bounded)
    assert default_candidates(_vdp(algorithm="tsit5")) == list(DEFAULT_CANDIDATES)
