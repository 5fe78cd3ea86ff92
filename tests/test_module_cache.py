"""Loaded modules are kept by source, compile options and device: solvers
that differ only in an option the source does not show run their own cubin
(CPU, with a stand-in for the loaded module)."""

import numpy as np

VDP = ["dx = y", "dy = mu * (1 - x**2) * y - x"]


def test_options_get_modules_of_their_own(monkeypatch):
    from cubie_b200 import Solver, _native, create_ODE_system, solver as solver_module
    monkeypatch.setattr(_native, "Module", lambda cubin, device, log: object())
    monkeypatch.setattr(solver_module, "_MODULE_CACHE", {})
    compiled = []

    def compile_cubin(source, options, use_cache=True):
        compiled.append(tuple(options))
        return b"cubin", ""

    monkeypatch.setattr(_native, "compile_cubin", compile_cubin)

    def module(**kw):
        sysm = create_ODE_system(VDP, states=["x", "y"], parameters=["mu"], precision=np.float32)
        return Solver(sysm, algorithm="radau", output_types=["state"], **kw).prepare(2.0)["module"]

    plain, exact, capped = module(), module(fast_math=False), module(max_registers=64)
    assert len({id(plain), id(exact), id(capped)}) == 3
    assert len(compiled) == 3
    assert "--use_fast_math" in compiled[0] and "--use_fast_math" not in compiled[1]
    assert "--maxrregcount=64" in compiled[2]
    # the same configuration again: the loaded module, nothing compiled
    assert module() is plain and module(fast_math=False) is exact and module(max_registers=64) is capped
    assert len(compiled) == 3
