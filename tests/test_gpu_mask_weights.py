"""A 2-D wet mask with values between 0 and 1, which the barotropic mode takes as
weights: every choice of its kernels gives the oracle's step (1e-5 in relative
L2, the bound of the other one-step checks)."""
import dataclasses

import numpy as np
import pytest

from oracle import step as ostep
from tests.gpu_util import build_pair, rel_l2, run_steps
from tests.test_gpu_dry_points import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["auto", "resident", "streaming"])
def test_one_step(kernel):
    grid, phys, dt, opts, st = _case(96, 40, 12, "islands")
    rng = np.random.default_rng(1)
    w = np.array(grid.wet_mask)
    w[(rng.random(w.shape) < 0.2) & (w > 0.5)] = 0.5
    grid = dataclasses.replace(grid, wet_mask=w)
    gpu, p = build_pair(grid, phys, dt, dict(opts, barotropic_kernel=kernel))
    got, want = run_steps(gpu, st, 1), ostep.step(st, p)
    wet = np.asarray(grid.wet_mask_3d)
    assert rel_l2(got["eta"], want["eta"]) < 1e-5
    for k in ("u", "v", "T", "S"):
        assert rel_l2(got[k], want[k], wet) < 1e-5, k
