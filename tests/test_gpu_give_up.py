"""Steps whose kernels gave up waiting for one another: the poll limit is set to
zero, so that the first word or barrier that is not there yet ends the wait.
Every block returns, the status names the timeout, and a reloaded state runs as
on a fresh handle: no word or barrier count of the broken launch is taken."""
import ctypes

import numpy as np
import pytest

from zhenmode_b200 import JaxStateG, _native, make_solver_global, workloads

pytestmark = pytest.mark.gpu


def _make(nx, ny, nz, land_lat, **extra):
    import torch
    grid = workloads.build_grid(nx, ny, nz, land_lat=land_lat)
    kw = dict(workloads.PLAIN_OPTIONS, forcing=workloads.wind_forcing(grid), dt_bt=75.0, dtype="float32", **extra)
    step, init, _ = make_solver_global(grid, workloads.PLAIN_PHYSICS, 1800.0, **kw)
    st = init(*workloads.initial_fields(grid))
    wet = torch.as_tensor(np.asarray(grid.wet_mask_3d, np.float32), device="cuda")
    g = torch.Generator(device="cuda").manual_seed(nx)
    rn = lambda: 0.05 * torch.randn(st.u.shape, generator=g, device="cuda") * wet  # noqa: E731
    return step, [JaxStateG(rn(), rn(), st.T + rn(), st.S, st.eta, st.ice) for _ in range(2)]


def _status(step):
    sv, code = step.solver, ctypes.c_int32()
    return sv.lib.zm_status(sv.handle, ctypes.byref(code))


@pytest.mark.parametrize("nx,ny,nz,land_lat,extra", [
    (96, 48, 6, 65.0, {}),                                                     # words between neighbours
    (96, 48, 6, 90.0, {}),                                                     # and the polar cap's barriers
    (96, 48, 6, 65.0, dict(sponge_days=5.0, sponge_cells=8)),                  # and the sums over the grid
    (96, 48, 6, 65.0, dict(project_adv_vel=True, projection_niter=20)),        # the projection, resident
    (1000, 400, 3, 65.0, dict(project_adv_vel=True, projection_niter=5)),      # and streamed
])
def test_a_reloaded_state_runs_as_on_a_fresh_handle(nx, ny, nz, land_lat, extra):
    import torch
    step, (first, second) = _make(nx, ny, nz, land_lat, **extra)
    sv = step.solver
    step(first)
    assert _status(step) == _native.ZM_OK
    sv.check(sv.lib.zm_set_wait_limit(sv.handle, 0), "zm_set_wait_limit")
    step(first)
    assert _status(step) == _native.ZM_ERR_TIMEOUT
    sv.check(sv.lib.zm_set_wait_limit(sv.handle, -1), "zm_set_wait_limit")
    got = step(second)
    assert _status(step) == _native.ZM_OK
    want = _make(nx, ny, nz, land_lat, **extra)[0](second)
    for k in ("u", "v", "T", "S", "eta"):
        assert torch.equal(getattr(got, k), getattr(want, k)), k


@pytest.mark.parametrize("extra", [{}, dict(project_adv_vel=True, projection_niter=20)])
@pytest.mark.parametrize("call", ["host", "ledger", "stage"])
def test_every_call_that_loads_a_state_starts_afresh(extra, call):
    """The host step, the ledger step and a stage after a step that gave up."""
    import torch
    from tests.gpu_util import FIELDS, run_stage
    from zhenmode_b200.ledger import make_budget_step

    def run(step, st):
        if call == "host":
            return step.advance(JaxStateG(*[t.cpu().numpy() for t in st[:5]], 0.0), 2)[:5]
        if call == "ledger":
            return [t.cpu().numpy() for t in make_budget_step(step)(st)[0][:5]]
        out = run_stage(step, 3, {k: getattr(st, k).double().cpu().numpy() for k in FIELDS})
        return [out[k] for k in FIELDS]

    step, (first, second) = _make(180, 90, 5, 65.0, **extra)
    sv = step.solver
    sv.check(sv.lib.zm_set_wait_limit(sv.handle, 0), "zm_set_wait_limit")
    step(first)
    torch.cuda.synchronize()
    sv.check(sv.lib.zm_set_wait_limit(sv.handle, -1), "zm_set_wait_limit")
    got = run(step, second)
    assert _status(step) == _native.ZM_OK
    for a, b in zip(got, run(_make(180, 90, 5, 65.0, **extra)[0], second)):
        assert np.array_equal(a, b)
