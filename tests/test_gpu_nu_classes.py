"""The strip classes of the nu_h kernel: every launch shape has its own class
table."""
import ctypes

import numpy as np
import pytest

from zhenmode_b200 import JaxStateG, make_solver_global, workloads
from zhenmode_b200.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def _member(seed):
    grid, physics, dt, kw, T, S = workloads.make_case("plain", 192, 96, 10, dtype="float32")
    step, init, _ = make_solver_global(grid, physics, dt, **dict(kw, nu_nsub=3))
    rng = np.random.default_rng(seed)
    st = init(T, S)
    import torch
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
    shape = lambda: [int(x) for x in info()]  # noqa: E731

    def info():
        sv = members[0][0].solver
        out = (ctypes.c_int32 * 16)()
        sv.check(sv.lib.zm_info(sv.handle, out, 16), "zm_info")
        return out[9], out[15]

    before = shape()
    sv = members[0][0].solver
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
