"""The strip classes of the nu_h kernel: strips with every face open take
another form of the update than the others, and every launch shape has its own
class table."""
import ctypes
import dataclasses

import numpy as np
import pytest

from tests.gpu_util import f32, run_stage
from zhenmode_b200 import JaxStateG, make_solver_global, workloads
from zhenmode_b200.ensemble import Ensemble

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(192, 96), (75, 47)])
def test_open_and_gated_strips_give_the_same_bits(nx, ny):
    """One dry column turns the open strips around it into gated ones.  Cells
    further from it than the stencils reach (3 subcycles, the finish's two
    cells) have the same inputs and coefficients in both runs; both forms add
    the same products in the same order, so the results are equal."""
    nz, i0, j0 = 4, nx // 2, ny // 2
    rng = np.random.default_rng(nx)
    out = []
    for island in (False, True):
        depth = np.full((nx, ny), 4900.0)
        depth[:, :3] = depth[:, -3:] = 0.0
        if island:
            depth[i0, j0] = 0.0
        grid = workloads.build_grid(nx, ny, nz, depth=depth)
        phys = dataclasses.replace(workloads.PLAIN_PHYSICS, nu_h=1.0e6)
        kw = dict(workloads.PLAIN_OPTIONS, forcing=workloads.wind_forcing(grid), dt_bt=75.0, nu_nsub=3,
                  dtype="float32")
        if not out:
            T, S = workloads.initial_fields(grid)
            state = f32(dict(u=rng.standard_normal((nx, ny, nz)), v=rng.standard_normal((nx, ny, nz)), T=T, S=S,
                             eta=np.zeros((nx, ny))))
        out.append(run_stage(make_solver_global(grid, phys, 1800.0, **kw)[0], 1, state))
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
    far = np.maximum(np.minimum(abs(i - i0), nx - abs(i - i0)), abs(j - j0)) > 6
    for k in ("u", "v"):
        assert np.array_equal(out[0][k][far], out[1][k][far]), k


def _member(seed):
    import torch
    grid, physics, dt, kw, T, S = workloads.make_case("plain", 192, 96, 10, dtype="float32")
    step, init, _ = make_solver_global(grid, physics, dt, **dict(kw, nu_nsub=3))
    rng = np.random.default_rng(seed)
    st = init(T, S)
    wet = torch.as_tensor(np.asarray(grid.wet_mask_3d, np.float32), device="cuda")
    move = lambda: 0.1 * torch.as_tensor(rng.standard_normal(st.u.shape), dtype=torch.float32, device="cuda") * wet  # noqa: E731
    return step, JaxStateG(move(), move(), st.T, st.S, st.eta, st.ice)


def test_tuning_a_member_leaves_the_ensembles_steps_right():
    """An ensemble's captured steps keep the launch shape they were captured
    with; tuning a member afterwards picks another shape (three subcycles fit a
    halo of three) and the ensemble's results stay those of untuned members."""
    import torch
    members = [_member(q) for q in range(2)]
    ens = Ensemble([m[0] for m in members])
    ens.load([m[1] for m in members])
    ens.advance(2)
    want = ens.store()
    sv = members[0][0].solver

    def shape():
        out = (ctypes.c_int32 * 16)()
        sv.check(sv.lib.zm_info(sv.handle, out, 16), "zm_info")
        return out[9], out[15]

    before = shape()
    sv.check(sv.lib.zm_autotune(sv.handle, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), None, None),
             "zm_autotune")
    if shape() == before:
        pytest.skip("the tuner kept the shape")
    members[0][0].advance(members[0][1], 0)  # the member has its own graphs again
    ens.load([m[1] for m in members])
    ens.advance(2)
    for a, b in zip(ens.store(), want):
        for k in ("u", "v", "T", "S", "eta"):
            assert torch.equal(getattr(a, k), getattr(b, k)), k
