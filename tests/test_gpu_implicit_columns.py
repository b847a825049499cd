"""The implicit vertical solve over column lengths from one level to all 64,
on grids that leave a partial warp, against the float64 oracle's linear stage:
1e-5 in relative L2 over the wet points, the bound of the other one-stage checks."""
import numpy as np
import pytest

from oracle import step as ostep
from tests.gpu_util import build_pair, rel_l2, run_stage
from tests.test_gpu_dry_points import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,shape", [("islands", (81, 30, 64)), ("all", (50, 22, 63)), ("islands", (100, 31, 33)),
                                        ("islands", (64, 24, 3)), ("none", (48, 21, 5))])
def test_linear_stage(kind, shape):
    import dataclasses
    grid, phys, dt, opts, st = _case(*shape, kind, vertical_diffusion="implicit")
    if kind == "islands":   # every column length
        wet3 = np.array(grid.wet_mask_3d)
        for i in range(shape[0]):
            wet3[i, 12, i % shape[2] + 1:] = 0.0
        grid = dataclasses.replace(grid, wet_mask_3d=wet3)
    gpu, p = build_pair(grid, phys, dt, opts)
    got = run_stage(gpu, 1, st)
    want = ostep.linear_half_step(st, p, dt / 2)
    wet = np.asarray(grid.wet_mask_3d)
    for k in ("u", "v", "T", "S"):
        if kind == "none":
            continue
        assert rel_l2(got[k], want[k], wet) < 1e-5, (k, rel_l2(got[k], want[k], wet))
    again = run_stage(gpu, 1, st)
    assert all(np.array_equal(got[k], again[k]) for k in got)


def test_no_diffusivity_leaves_the_explicit_forms_bits():
    """With nu_v = kappa_v = 0 the solve is the identity, exactly, and the linear
    stage differs from the explicit form in nothing: the same bits."""
    import dataclasses
    nx, ny, nz = 75, 31, 14
    out = []
    for extra in ({}, {"vertical_diffusion": "implicit"}):
        grid, phys, dt, opts, st = _case(nx, ny, nz, "islands", **extra)
        gpu, _ = build_pair(grid, dataclasses.replace(phys, nu_v=0.0, kappa_v=0.0), dt, opts)
        out.append(run_stage(gpu, 1, st))
    for k in ("u", "v", "T", "S"):
        assert np.array_equal(out[0][k], out[1][k]), k
