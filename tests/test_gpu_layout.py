"""The layout change between the caller's (nx, ny, nz) arrays and the internal
fields at the edges of its tiles, the classification a step makes of its own
result, and the tracer-term and budget diagnostics on grids that end inside a
tile and on columns with dry levels between wet ones."""
import ctypes

import numpy as np
import pytest

from oracle import budgets as obudgets
from oracle import step as ostep
from tests import gpu_util as gu
from tests.test_gpu_dry_points import _case
from zhenmode_b200 import JaxStateG, _native, make_solver_global, workloads

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


@pytest.mark.parametrize("kind,shape,extra", [
    ("islands", (96, 40, 12), {}), ("holes", (75, 31, 27), {}), ("all", (100, 46, 37), {"fct_adv": False}),
    ("holes", (64, 45, 64), {"fct_adv": False, "monotone_adv": False, "conservative_kv": True}),
    ("islands", (50, 22, 3), {"localize_conv": False}), ("none", (48, 21, 5), {})])
def test_tracer_terms_at_the_edges(kind, shape, extra):
    """float32 difference operators of O(1) anomalies: 1e-5 in relative L2, as the other stage checks;
    columns with an interface whose stability margin is within float32 rounding are left out of the
    convective term.  Where dry levels interrupt a column the flux divergence of a constant does not
    cancel, so the advection of an anomaly is not that of T: it is left out there."""
    from oracle import params as oparams
    grid, phys, dt, opts, st = _case(*shape, kind, **extra)
    out = make_solver_global(grid, phys, dt, return_params=True, **dict(opts, dtype="float32"))
    p = oparams.build_params(grid, phys, dt, **dict({k: v for k, v in opts.items() if k in oparams.SUPPORTED},
                                                    dtype="float64"))
    got = out[4](JaxStateG(*gu.to_device(st), 0.0)).double().cpu().numpy()
    want = ostep.tracer_terms(st, p)
    margin = np.abs(7.6e-4 * np.diff(st["S"], axis=2) - 2.0e-4 * np.diff(st["T"], axis=2)).min(axis=2) > 1e-7
    for n, name in enumerate(("adv", "diff_h", "diff_v", "conv", "gm", "redi")):
        if kind == "holes" and name == "adv":
            continue
        a, b = (got[n][margin], want[n][margin]) if name == "conv" else (got[n], want[n])
        if np.abs(b).max() == 0:
            assert np.abs(a).max() == 0, name
        else:
            assert gu.rel_l2(a, b) < 1e-5, (name, gu.rel_l2(a, b))


@pytest.mark.parametrize("kind,shape", [("islands", (50, 22, 3)), ("holes", (100, 46, 33)), ("all", (64, 45, 64)),
                                        ("islands", (160, 64, 32)), ("holes", (200, 100, 31))])
def test_budgets_at_the_edges(kind, shape):
    """Compensated float64 sums: 1e-12 of the oracle's, for column counts that leave a remainder."""
    grid, phys, dt, opts, st = _case(*shape, kind)
    step = make_solver_global(grid, phys, dt, **dict(opts, dtype="float32"))[0]
    T32, S32 = (np.asarray(st[k], np.float32) for k in "TS")
    got = step.budget_diagnostics(JaxStateG(*gu.to_device(st), None)).as_dict()
    want = obudgets.budget_diagnostics(T32, S32, grid.dx_2d, grid.dy, grid.z, grid.wet_mask, grid.wet_mask_3d)
    for name in obudgets.FIELDS:
        assert abs(got[name] - want[name]) <= 1e-12 * abs(want[name]), (name, got[name], want[name])
