"""Columns with dry levels between wet ones, and dry surfaces over wet water,
against the float64 oracle in the stages that skip dry levels.

The step holds T and S as anomalies from (T_ref, S_ref); where an interface is
closed inside a column the flux of the constant part does not cancel, so the
nonlinear stage is compared with T_ref = S_ref = 0, where both sides advect the
same numbers.  The implicit solve takes columns with a wet surface and passes the
others through; it is compared on the former (a column's solve reads no other)."""
import dataclasses

import numpy as np
import pytest

from oracle import step as ostep
from tests.gpu_util import build_pair, rel_l2, run_stage, run_steps
from tests.test_gpu_dry_points import _case

pytestmark = pytest.mark.gpu

TOL = 1e-5  # of the other one-step checks


@pytest.mark.parametrize("shape", [(96, 40, 12), (75, 31, 27)])
@pytest.mark.parametrize("extra", [{}, {"conservative_kv": True, "fct_adv": False}, {"localize_conv": False}])
def test_nonlinear_stage_and_step(shape, extra):
    grid, phys, dt, opts, st = _case(*shape, "holes", **{k: v for k, v in extra.items() if k != "localize_conv"})
    opts.update(extra)
    gpu, p = build_pair(grid, dataclasses.replace(phys, T_ref=0.0, S_ref=0.0), dt, opts)
    wet = np.asarray(grid.wet_mask_3d)
    for got, want in ((run_stage(gpu, 2, st), ostep.explicit_full_step(st, p)),
                      (run_steps(gpu, st, 1), ostep.step(st, p))):
        for k in ("u", "v", "T", "S"):
            assert rel_l2(got[k], want[k], wet) < TOL, (k, rel_l2(got[k], want[k], wet))


@pytest.mark.parametrize("shape", [(96, 40, 12), (75, 31, 27)])
def test_implicit_columns(shape):
    grid, phys, dt, opts, st = _case(*shape, "holes", vertical_diffusion="implicit")
    phys = dataclasses.replace(phys, nu_v=1.0e-2, kappa_v=1.0e-3)
    gpu, p = build_pair(grid, phys, dt, opts)
    wet = np.asarray(grid.wet_mask_3d)
    solved = wet * (wet[:, :, :1] > 0.5)
    assert 0.0 < solved.sum() < wet.sum()
    got, want = run_stage(gpu, 1, st), ostep.linear_half_step(st, p, dt / 2)
    for k in ("u", "v", "T", "S"):
        assert rel_l2(got[k], want[k], solved) < TOL, (k, rel_l2(got[k], want[k], solved))
