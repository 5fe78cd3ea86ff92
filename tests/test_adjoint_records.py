"""The adjoint's record form (a record of every accepted step, nothing
replayed) against its checkpoint form: the records are the replay's own, so
statuses and step limits are the same and the gradients agree to the
roundings a separately compiled kernel may contract differently."""

import ctypes
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent / "host_emu"))

FHN = ["dV = V - V**3 / 3 - w + I", "dw = (V + a - b * w) / tau"]
VDP = ["dx = y", "dy = mu * (1 - x**2) * y - x"]
DRIVER = r"""
extern "C" void emu_records(cbx_solve_args* a, cbx_adjoint_args* g, int phase, int block) {
    blockDim = {(unsigned)block, 1, 1};
    gridDim = {1, 1, 1};
    blockIdx = {0, 0, 0};
    for (int t = 0; t < block; ++t) {
        threadIdx = {(unsigned)t, 0, 0};
        if (phase == 0) cbx_adjoint_forward_records(*a, *g);
        else if (phase == 1) cbx_adjoint_backward_records(*a, *g);
        else if (phase == 2) cbx_adjoint_forward_pairs(*a, *g);
        else cbx_adjoint_backward_pairs(*a, *g);
    }
}
"""


def _solver(name, precision=np.float32, mixed=True):
    from cubie_b200 import Solver, create_ODE_system
    kw = dict(rtol=1e-5, atol=1e-5, output_types=["state"], save_every=1.0, adjoint=True, mixed_precision=mixed)
    if name == "fhn":
        sysm = create_ODE_system(FHN, states=["V", "w"], parameters=["a", "b", "tau", "I"], precision=precision)
        return Solver(sysm, algorithm="dormand-prince-54", **kw)
    sysm = create_ODE_system(VDP, states=["x", "y"], parameters=["mu"], precision=precision)
    return Solver(sysm, algorithm="ros3p", linear_correction_type="direct", preconditioner_type=None, **kw)


def _batch(name, n, seed=0):
    rng = np.random.default_rng(seed)
    if name == "fhn":
        return (np.stack([rng.uniform(1, 2, n), rng.uniform(-0.5, 0.5, n)]),
                np.stack([rng.uniform(0.6, 0.8, n), rng.uniform(0.7, 0.9, n), rng.uniform(8, 13, n),
                          rng.uniform(0.5, 0.7, n)]))
    return np.stack([rng.uniform(1, 2, n), rng.uniform(-1, 1, n)]), rng.uniform(0.5, 3.0, (1, n))


def _emulated_against_replay(name, every, ckpts, pairs=False):
    """Both forms in emulation: the same bits; returns (steps, statuses)."""
    from emu import compile_emulated, run_emulated_adjoint
    from cubie_b200 import _native
    s = _solver(name)
    x0, p = _batch(name, 5)
    T = 6.0
    state, status, gi, gp = run_emulated_adjoint(s, x0, p, T, lambda y: 0.1 * y, every, ckpts)
    prep = s.prepare(T, 0.0, 0.0, None, None, load=False)
    lib = compile_emulated(prep["gen"].source + DRIVER)
    n, cap = x0.shape[1], every * ckpts
    lanes = n + 3 if pairs else n
    x, q = np.ascontiguousarray(x0, np.float32), np.ascontiguousarray(p, np.float32)
    out = dict(state=np.zeros_like(state), status=np.zeros_like(status), work=np.zeros(2, np.uint64),
               seg=np.full(lanes * cap * int(lib.emu_record_bytes()) // 8 + 2, np.nan), count=np.zeros(n, np.int32),
               steps=np.zeros(n, np.int32), gi=np.zeros_like(gi), gp=np.zeros((p.shape[0], n), np.float32))
    grad = np.ascontiguousarray(0.1 * state, np.float32)
    a = _native.SolveArgs()
    a.inits, a.params, a.state_out = x.ctypes.data, q.ctypes.data, out["state"].ctypes.data
    a.status_out, a.work_counter = out["status"].ctypes.data, out["work"].ctypes.data
    a.n_runs = a.run_stride = n
    a.duration, a.save_stop, a.summary_stop = T, float(prep["save_stop"]), float(prep["summary_stop"])
    a.n_save_rows = int(prep["n_save"])
    g = _native.AdjointArgs()
    g.seg, g.ckpt_count, g.step_count = (out[k].ctypes.data for k in ("seg", "count", "steps"))
    g.ckpt_every, g.max_ckpts = every, ckpts
    g.lane_words = lanes
    g.grad_state, g.grad_inits, g.grad_params = grad.ctypes.data, out["gi"].ctypes.data, out["gp"].ctypes.data
    lib.emu_records(ctypes.byref(a), ctypes.byref(g), 2 if pairs else 0, 32)
    out["work"][:] = 0
    lib.emu_records(ctypes.byref(a), ctypes.byref(g), 3 if pairs else 1, 32)
    # one compiler, no contraction: the same bits
    np.testing.assert_array_equal(out["state"], state)
    np.testing.assert_array_equal(out["status"], status)
    np.testing.assert_array_equal(out["gi"], gi)
    np.testing.assert_array_equal(out["gp"], gp)
    assert np.all(np.isnan(out["seg"][-2:]))          # nothing past the records
    return out["steps"], status


@pytest.mark.parametrize("name", ["fhn", "vdp"])
def test_emulated_records_equal_replay(name):
    steps, _ = _emulated_against_replay(name, 4, 64)
    assert steps.min() > 2 * 4


# records in pairs of steps (an even limit of steps); runs that stop at the
# limit and runs that end before it
@pytest.mark.parametrize("name", ["fhn", "vdp"])
@pytest.mark.parametrize("every,ckpts", [(4, 32), (3, 4), (1, 2), (7, 2)])
def test_emulated_pairs_equal_replay(name, every, ckpts):
    steps, status = _emulated_against_replay(name, every, ckpts, pairs=True)
    if every * ckpts <= 15:
        assert np.all(steps == every * ckpts) and np.all(status == 32)
    else:
        assert steps.min() > 2 * every


@pytest.mark.gpu
@pytest.mark.parametrize("name,precision,mixed", [("fhn", np.float32, True), ("vdp", np.float32, True),
                                                  ("fhn", np.float64, False)])
@pytest.mark.parametrize("n", [65536, 65537])
@pytest.mark.parametrize("every,ckpts", [(64, 16), (3, 5)])
def test_record_layouts_equal_checkpoints_run_by_run(cuda_device, name, precision, mixed, n, every, ckpts):
    """Both record layouts against checkpoints, every run by itself: states,
    statuses and gradients, with a tolerance scale per run."""
    import torch
    from cubie_b200.adjoint import AdjointIntegrator
    s = _solver(name, precision, mixed)
    x0, p = (torch.tensor(v.astype(precision), device="cuda") for v in _batch(name, n, 3))
    scale = torch.tensor(10.0 ** np.random.default_rng(4).uniform(-0.5, 0.5, n), device="cuda")
    out = []
    for share in (0.125, 0.0):
        integ = AdjointIntegrator(s, ckpt_every=every, max_ckpts=ckpts, record_share=share)
        state, status, saved = integ.forward(x0, p, 8.0, tol_scale=scale)
        assert (saved["records"] is not None) == (share > 0)
        out.append((state.clone(), status.clone(), *integ.backward(saved, 0.1 * state)))
    (sa, ta, ga, pa), (sb, tb, gb, pb) = out
    assert torch.equal(ta, tb) and bool((ta != 0).any()) == (every == 3)
    # as in test_records_equal_checkpoints, each run against its own size
    tol = 100 * 200 * (1.2e-7 if precision == np.float32 else 2.3e-16)
    for u, v in ((sa, sb), (ga, gb), (pa, pb)):
        u, v = u.reshape(-1, n).double(), v.reshape(-1, n).double()
        assert float(((u - v).norm(dim=0) / v.norm(dim=0).clamp(min=1e-3)).max()) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("name,precision,mixed,n", [("fhn", np.float32, True, 1001), ("fhn", np.float64, False, 33),
                                                    ("vdp", np.float32, True, 1), ("vdp", np.float32, True, 777),
                                                    ("fhn", np.float32, True, 151553)])   # more runs than lanes
@pytest.mark.parametrize("every,ckpts", [(64, 64), (7, 90), (3, 4)])
def test_records_equal_checkpoints(cuda_device, name, precision, mixed, n, every, ckpts):
    import torch
    from cubie_b200.adjoint import AdjointIntegrator
    s = _solver(name, precision, mixed)
    x0, p = (torch.tensor(v.astype(precision), device="cuda") for v in _batch(name, n, 3))
    out = []
    for share in (0.125, 0.0):
        integ = AdjointIntegrator(s, ckpt_every=every, max_ckpts=ckpts, record_share=share)
        state, status, saved = integ.forward(x0, p, 8.0)
        assert (saved["records"] is not None) == (share > 0 and n < 151553)
        out.append((state.clone(), status.clone(), *integ.backward(saved, 0.1 * state)))
    (sa, ta, ga, pa), (sb, tb, gb, pb) = out
    assert torch.equal(ta, tb)
    if every * ckpts == 12:
        assert bool((ta != 0).any())          # runs that reach the step limit stop alike
    # the step is one function in both kernels; a contraction chosen
    # differently is a rounding per operation, amplified over some hundred
    # steps by the flow's own sensitivity (below 100 on these windows)
    tol = 100 * 200 * (1.2e-7 if precision == np.float32 else 2.3e-16)
    for u, v in ((sa, sb), (ga, gb), (pa, pb)):
        assert float((u - v).norm()) <= tol * float(v.norm())


@pytest.mark.gpu
@pytest.mark.parametrize("name,precision,mixed", [("fhn", np.float32, True), ("fhn", np.float64, False),
                                                  ("vdp", np.float32, True)])
def test_records_while_every_run_has_a_lane(cuda_device, name, precision, mixed):
    """The record form ends at the runs its kernels hold at once, which their
    registers decide (FP64 takes twice as many)."""
    import torch
    from cubie_b200.adjoint import AdjointIntegrator
    s = _solver(name, precision, mixed)
    integ = AdjointIntegrator(s, ckpt_every=3, max_ckpts=4)
    x0, p = (torch.tensor(v.astype(precision), device="cuda") for v in _batch(name, 2, 3))
    _, _, saved = integ.forward(x0, p, 0.5)
    lanes = saved["prep"]["record_lanes"]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert lanes % (sms * s.block_size) == 0 and 256 <= lanes // sms <= 2048
    assert lanes // sms <= (640 if precision == np.float64 else 1280)      # 96 and 48 registers
    for n in (lanes, lanes + 1):
        x, q = x0[:, :1].repeat(1, n), p[:, :1].repeat(1, n)
        state, status, saved = integ.forward(x, q, 0.5)
        assert (saved["records"] is not None) == (n == lanes)
        gi, gp = integ.backward(saved, torch.ones_like(state))
        assert torch.equal(gi, gi[:, :1].expand_as(gi)) and torch.equal(gp, gp[:, :1].expand_as(gp))


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["fhn", "vdp"])
@pytest.mark.parametrize("share", [0.125, 0.0])
def test_inputs_written_between_forward_and_backward(cuda_device, name, share):
    """The gradient is the forward pass's, whatever the caller writes to the
    initial values, parameters and tolerance scales after it."""
    import torch
    from cubie_b200.adjoint import AdjointIntegrator
    s = _solver(name)
    out = []
    for write in (False, True):
        x0, p = (torch.tensor(v.astype(np.float32), device="cuda") for v in _batch(name, 300, 3))
        scale = torch.ones(300, dtype=torch.float64, device="cuda")
        integ = AdjointIntegrator(s, record_share=share)
        state, _, saved = integ.forward(x0, p, 4.0, tol_scale=scale)
        if write:
            x0.fill_(7.0), p.mul_(1.5), scale.fill_(1e-3)
        out.append(integ.backward(saved, 0.1 * state))
    for a, b in zip(*out):
        assert torch.equal(a, b)


@pytest.mark.gpu
def test_records_leave_room_for_the_caller(cuda_device, monkeypatch):
    """Large records need four times their size besides torch's tensors; the
    answer stays with the integrator and the size."""
    import torch
    from cubie_b200 import adjoint
    s = _solver("fhn")
    x0, p = (torch.tensor(v.astype(np.float32), device="cuda") for v in _batch("fhn", 64, 3))
    nbytes = 64 * 64 * 64 * 16
    free = []
    monkeypatch.setattr(adjoint, "RECORDS_UNASKED", 0)
    monkeypatch.setattr(adjoint, "_free_bytes", lambda dev: free.pop())
    for room in (4 * nbytes, 4 * nbytes - 1):
        free.append(room)
        integ = adjoint.AdjointIntegrator(s)
        for _ in range(3):
            _, _, saved = integ.forward(x0, p, 2.0)
            assert (saved["records"] is not None) == (room == 4 * nbytes)
        assert not free
    monkeypatch.setattr(adjoint, "RECORDS_UNASKED", nbytes)          # small records are not asked for
    _, _, saved = adjoint.AdjointIntegrator(s).forward(x0, p, 2.0)
    assert saved["records"] is not None


@pytest.mark.gpu
def test_modules_without_record_kernels_use_checkpoints(cuda_device):
    """A cubin saved before there were record kernels: its checkpoint launches
    run, a record launch is refused, the integrator takes checkpoints."""
    import re
    import torch
    from cubie_b200 import _native
    from cubie_b200.adjoint import AdjointIntegrator
    s = _solver("fhn")
    x0, p = (torch.tensor(v.astype(np.float32), device="cuda") for v in _batch("fhn", 40, 3))
    want = AdjointIntegrator(s, record_share=0.0)
    state, _, saved = want.forward(x0, p, 4.0)
    grads = want.backward(saved, state)
    prep = dict(saved["prep"])
    header = (_native.DEVICE_INCLUDE / "cbx_adjoint.cuh").read_text()
    macro = header[header.index("#define CBX_DEFINE_ADJOINT_KERNELS(CFG)"):]
    first = macro[:macro.index('    extern "C" __global__ void CBX_LAUNCH_BOUNDS(CFG) cbx_adjoint_forward_records')]
    first = first.rstrip().rstrip("\\").replace("ADJOINT_KERNELS", "TWO_ADJOINT_KERNELS", 1)
    source, n = re.subn(r"CBX_DEFINE_ADJOINT_KERNELS\((.*)\)", lambda m: first + f"\nCBX_DEFINE_TWO_ADJOINT_KERNELS({m[1]})",
                        prep["gen"].source)
    assert n == 1
    cubin, log = _native.compile_cubin(source, _native.default_options())
    old = _native.Module(cubin, 0, log)
    assert old.adjoint_lanes(128) == 0
    key = next(k for k, v in s._prepared.items() if v is saved["prep"])
    s._prepared[key] = dict(saved["prep"], module=old)
    s._prepared[key].pop("record_lanes", None)
    integ = AdjointIntegrator(s)
    state2, _, saved2 = integ.forward(x0, p, 4.0)
    assert saved2["records"] is None
    for a, b in zip((state, *grads), (state2, *integ.backward(saved2, state))):
        assert torch.equal(a, b)
    adj = _native.AdjointArgs()
    buf = torch.zeros((1 << 16,), device="cuda", dtype=torch.int32)
    adj.seg = adj.ckpt_count = adj.step_count = buf.data_ptr()
    adj.lane_words, adj.ckpt_every, adj.max_ckpts = 40, 1, 2
    args = s.make_args(s._prepared[key], saved2["bufs"], x0, p, None, 40, 4.0, 0.0, 0.0)
    with pytest.raises(_native.NativeError, match="without the record kernels"):
        old.adjoint_launch(args, adj, 0, 128, records=True)


@pytest.mark.gpu
def test_free_bytes_follow_the_tensors(cuda_device):
    import torch
    from cubie_b200.adjoint import _free_bytes
    total = torch.cuda.get_device_properties(0).total_memory
    before = _free_bytes(0)
    big = torch.empty((1 << 28,), dtype=torch.uint8, device="cuda")
    assert before - _free_bytes(0) == big.numel() and before <= total
    del big
    assert _free_bytes(0) == before


@pytest.mark.gpu
def test_autograd_passes_release_their_records(cuda_device):
    import gc
    import torch
    from cubie_b200.adjoint import AdjointIntegrator, solve_ivp_adjoint
    s = _solver("fhn")
    x0, p = (torch.tensor(v.astype(np.float32), device="cuda") for v in _batch("fhn", 500, 3))
    integ = AdjointIntegrator(s, 64, 64)
    used = []
    gc.collect()
    gc.disable()
    try:
        for _ in range(3):
            q = p.clone().requires_grad_(True)
            state, status = solve_ivp_adjoint(s, x0.clone().requires_grad_(True), q, 8.0, integrator=integ)
            (state ** 2).mean().backward()
            assert bool(torch.isfinite(q.grad).all())
            del state, status, q
            used.append(torch.cuda.memory_allocated())
    finally:
        gc.enable()
    assert used[1] == used[0] and used[2] == used[0]
