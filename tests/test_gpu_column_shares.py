"""The nonlinear and linear stages where the split of a column's levels between
threads and blocks leaves remainders: few levels, level counts that no share
divides, several convective substeps (one thread takes the column) and gates that
open whole columns.  1e-5 in relative L2 of the float64 oracle, as the other
one-stage checks."""
import dataclasses

import numpy as np
import pytest

from oracle import step as ostep
from tests.gpu_util import build_pair, rel_l2, run_stage
from tests.test_gpu_dry_points import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,shape", [("islands", (96, 40, 3)), ("all", (60, 25, 5)), ("islands", (160, 72, 21)),
                                        ("all", (96, 41, 63)), ("islands", (64, 33, 64))])
@pytest.mark.parametrize("kappa_conv,extra", [(None, {}), (0.1, {}), (0.1, {"localize_conv": False}),
                                              (0.01, {"localize_conv": False})])
def test_stages(kind, shape, kappa_conv, extra):
    grid, phys, dt, opts, st = _case(*shape, kind, **extra)
    if kappa_conv is not None:
        phys = dataclasses.replace(phys, kappa_conv=kappa_conv)
    gpu, p = build_pair(grid, phys, dt, opts)
    wet = np.asarray(grid.wet_mask_3d)
    for stage in (1, 2):
        got = run_stage(gpu, stage, st)
        want = ostep.linear_half_step(st, p, dt / 2) if stage == 1 else ostep.explicit_full_step(st, p)
        for k in ("u", "v", "T", "S"):
            assert rel_l2(got[k], want[k], wet) < 1e-5, (stage, k, rel_l2(got[k], want[k], wet))
