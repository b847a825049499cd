"""The layout change between the caller's (nx, ny, nz) arrays and the internal
fields at the edges of its tiles, and the classification a step makes of its own
result."""
import ctypes

import numpy as np
import pytest

from tests import gpu_util as gu
from zhenmode_b200 import _native, make_solver_global, workloads

pytestmark = pytest.mark.gpu


def _stream():
    import torch
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("nx,ny,nz", [(48, 24, 10), (32, 20, 3), (90, 45, 15), (100, 47, 37), (64, 21, 63),
                                      (50, 22, 64)])
def test_a_state_passes_through_unchanged(nx, ny, nz):
    """Zero steps: velocities and eta bit for bit, tracers as their anomaly rounds in float32."""
    import torch
    grid, physics, dt, kw, T, S = workloads.make_case("plain", nx, ny, nz, dtype="float32")
    solver = make_solver_global(grid, physics, dt, **kw)[0].solver
    rng = np.random.default_rng(nz)
    host = {k: rng.standard_normal((nx, ny, nz)).astype(np.float32) for k in "uvTS"}
    host["T"] += 10
    host["S"] += 35
    host["eta"] = rng.standard_normal((nx, ny)).astype(np.float32)
    fields = gu.to_device(host)
    outs = [torch.full_like(f, float("nan")) for f in fields]
    sin = _native.ZmState(*[t.data_ptr() for t in fields])
    sout = _native.ZmState(*[t.data_ptr() for t in outs])
    solver.check(solver.lib.zm_step(solver.handle, _stream(), ctypes.byref(sin), ctypes.byref(sout), 0), "zm_step")
    got = dict(zip(gu.FIELDS, [t.cpu().numpy() for t in outs]))
    for name in ("u", "v", "eta"):
        assert np.array_equal(got[name], host[name]), name
    for name, ref in (("T", physics.T_ref), ("S", physics.S_ref)):
        r = np.float32(ref)
        assert np.array_equal(got[name], (host[name] - r) + r), name


@pytest.mark.parametrize("edit", [
    lambda s: None,
    lambda s: s["T"].__setitem__((3, 4, 0), np.nan),
    lambda s: s["u"].__setitem__((0, 6, 2), 50.0),       # a dry point keeps it
    lambda s: s["v"].__setitem__((20, 12, 2), -500.0),
    lambda s: s["eta"].__setitem__((20, 12), 400.0),
    lambda s: s["eta"].__setitem__((0, 5), 20.0),
    lambda s: s["S"].__setitem__((0, 7, 9), np.inf),
])
@pytest.mark.parametrize("nsteps", [1, 2])
def test_a_step_classifies_its_result_as_the_pass_over_the_state_does(edit, nsteps):
    """The code after stepping equals that of loading the stepped state and taking no step."""
    import torch
    _, step, state, _ = _monitor_case()
    solver = step.solver
    state = {k: np.array(v, np.float32) for k, v in state.items()}
    edit(state)
    code = ctypes.c_int32(-1)

    def run(fields, n):
        outs = [torch.empty_like(f) for f in fields]
        sin = _native.ZmState(*[t.data_ptr() for t in fields])
        sout = _native.ZmState(*[t.data_ptr() for t in outs])
        solver.check(solver.lib.zm_step(solver.handle, _stream(), ctypes.byref(sin), ctypes.byref(sout), n), "zm_step")
        solver.check(solver.lib.zm_status(solver.handle, ctypes.byref(code)), "zm_status")
        return outs, int(code.value)

    outs, stepped = run(gu.to_device(state), nsteps)
    assert run(outs, 0)[1] == stepped
    good, ok = run(gu.to_device(_monitor_case()[2]), 1)   # nothing stays behind from the edited state
    assert ok == 0


_made = {}


def _monitor_case():
    if not _made:
        grid, physics, dt, kw, T, S = workloads.make_case("plain", 48, 24, 10, dtype="float32")
        from oracle.params import init_state
        gpu, p = gu.build_pair(grid, physics, dt, kw)
        _made["it"] = (grid, gpu, gu.f32(init_state(p, T, S)), p)
    return _made["it"]
