"""Masks on which the kernels leave out dry points: columns with dry levels
between wet ones, whole tiles and levels without a wet point, grids that end
inside a tile, and dry points that hold values of their own.  One step against
the float64 oracle at the bound of the other one-step checks (1e-5), the
dry points bit for bit, and the stages' pass-through of dry tracers.  Columns
with dry levels between wet ones are held to the oracle in the linear stage,
whose stencils read those levels."""
import dataclasses

import numpy as np
import pytest

from tests.gpu_util import build_pair, f32, rel_l2, run_stage, run_steps
from zhenmode_b200 import workloads as W
from oracle import step as ostep

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _case(nx, ny, nz, kind, **extra):
    rng = np.random.default_rng(nx * 7 + ny)
    depth = np.full((nx, ny), 4000.0)
    depth[:, :4] = 0.0
    depth[:, -3:] = 0.0
    if kind == "islands":   # whole column tiles dry, and shallow water beside deep water
        depth[nx // 3: nx // 3 + 40, :] = 0.0
        depth[:, ny // 2:] = np.where(depth[:, ny // 2:] > 0, 300.0, 0.0)
        depth[nx // 2, ny // 4] = 5000.0
    grid = W.build_grid(nx, ny, nz, depth=depth)
    wet3 = np.array(grid.wet_mask_3d)
    if kind == "holes":     # dry levels inside the column, dry tops over wet water, single wet points
        wet3 *= rng.random((nx, ny, nz)) < 0.9
        wet3[5:9, 6:10, 0] = 0.0
        wet3[10:50, 5:9, 2:] = 0.0
        wet3[20, 7, nz - 1] = 1.0
    if kind == "none":      # no wet point at all
        wet3[:] = 0.0
    if kind == "all":       # no dry point
        wet3[:] = 1.0
    wet2 = (wet3[:, :, 0] > 0.5).astype(np.float64)
    if kind == "holes":
        wet2 = (wet3.max(2) > 0.5).astype(np.float64)
    grid = dataclasses.replace(grid, wet_mask_3d=wet3, wet_mask=wet2, ocean_mask=wet2 > 0.5, land_mask=wet2 < 0.5)
    T, S = W.initial_fields(grid, perturb_sigma=0.3)
    st = dict(u=0.1 * rng.standard_normal((nx, ny, nz)), v=0.1 * rng.standard_normal((nx, ny, nz)),
              T=T + 0.3 * rng.standard_normal(T.shape), S=S, eta=0.1 * rng.standard_normal((nx, ny)) * wet2)
    opts = dict(W.PLAIN_OPTIONS, forcing=W.wind_forcing(grid), dt_bt=75.0, polar_cap_rows=2, polar_cap_taper=2,
                **extra)
    phys = dataclasses.replace(W.PLAIN_PHYSICS, nu_h=1.0e6)
    return grid, phys, 1800.0, opts, f32(st)


@pytest.mark.parametrize("kind", ["islands", "holes", "none", "all"])
@pytest.mark.parametrize("shape", [(96, 40, 12), (75, 31, 27)])
@pytest.mark.parametrize("extra", [{}, {"vertical_diffusion": "implicit"}, {"conservative_kv": True, "fct_adv": False}])
def test_one_step(kind, shape, extra):
    grid, phys, dt, opts, st = _case(*shape, kind, **extra)
    gpu, p = build_pair(grid, phys, dt, opts)
    got = run_steps(gpu, st, 1)
    want = ostep.step(st, p)
    wet = np.asarray(grid.wet_mask_3d)
    for k in ("u", "v", "T", "S"):
        if kind in ("islands", "all"):
            assert rel_l2(got[k], want[k], wet) < TOL, (k, rel_l2(got[k], want[k], wet))
        dry = wet < 0.5
        held = np.array(st[k])
        if k == "v":
            held[:, 0] = held[:, -1] = 0.0
        # T, S pass through the anomaly round trip of the boundary
        assert np.allclose(got[k][dry], held[dry], rtol=0, atol=0 if k in ("u", "v") else 4e-6), k
    if kind in ("islands", "all"):
        assert rel_l2(got["eta"], want["eta"]) < TOL
    again = run_steps(gpu, st, 1)
    for k in got:
        assert np.array_equal(got[k], again[k])


@pytest.mark.parametrize("kind,stages", [("islands", (1, 2)), ("holes", (1,))])
def test_stages_pass_dry_tracers(kind, stages):
    """The linear and nonlinear stages alone, whose results include the dry points."""
    grid, phys, dt, opts, st = _case(75, 31, 14, kind)
    gpu, p = build_pair(grid, phys, dt, opts)
    wet = np.asarray(grid.wet_mask_3d)
    for stage in stages:
        got = run_stage(gpu, stage, st)
        want = ostep.linear_half_step(st, p, dt / 2) if stage == 1 else ostep.explicit_full_step(st, p)
        for k in ("u", "v", "T", "S"):
            assert rel_l2(got[k], want[k]) < TOL, (stage, k, rel_l2(got[k], want[k]))
            assert rel_l2(got[k], want[k], wet) < TOL, (stage, k)


def test_diagnostics_of_a_broken_state_leave_the_step_clean():
    """Diagnostics and closure rows of a state full of NaN, then a step: the
    step's work fields hold nothing of them."""
    import torch
    from zhenmode_b200 import JaxStateG, make_solver_global
    grid, phys, dt, opts, st = _case(75, 31, 14, "islands")
    made = make_solver_global(grid, phys, dt, dtype="float32", return_params=True, **opts)
    step, diagnostics, terms = made[0], made[2], made[4]
    good = JaxStateG(*[torch.as_tensor(st[k].astype(np.float32), device="cuda") for k in ("u", "v", "T", "S", "eta")], 0.0)
    bad = JaxStateG(*[torch.full_like(t, float("nan")) for t in good[:5]], 0.0)
    want = step(good)
    diagnostics(bad)
    terms(bad)
    step.closure_features(bad)
    step(bad)
    got = step(good)
    for a, b in zip(got[:5], want[:5]):
        assert torch.equal(a, b)
