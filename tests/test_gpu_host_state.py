"""States in host memory: pageable arrays (staged by several threads),
pinned ones, unaligned ones and in-place results give what device states give."""
import ctypes

import numpy as np
import pytest

from tests import gpu_util as gu
from zhenmode_b200 import JaxStateG, _native, make_solver_global, workloads

pytestmark = pytest.mark.gpu


def _case(nx, ny, nz):
    grid, physics, dt, kw, T, S = workloads.make_case("plain", nx, ny, nz, dtype="float32")
    step = make_solver_global(grid, physics, dt, **kw)[0]
    rng = np.random.default_rng(nx)
    wet = np.asarray(grid.wet_mask_3d)
    st = dict(u=0.1 * rng.standard_normal(T.shape) * wet, v=0.1 * rng.standard_normal(T.shape) * wet,
              T=T + 0.1 * rng.standard_normal(T.shape) * wet, S=S, eta=np.zeros(T.shape[:2]))
    return step, {k: np.ascontiguousarray(v, dtype=np.float32) for k, v in st.items()}


def _host_step(step, ins, outs, n):
    sv = step.solver
    a = _native.ZmState(*[x.ctypes.data for x in ins])
    b = _native.ZmState(*[x.ctypes.data for x in outs])
    sv.check(sv.lib.zm_step_host(sv.handle, None, ctypes.byref(a), ctypes.byref(b), n), "zm_step_host")


@pytest.mark.parametrize("shape", [(32, 20, 4), (90, 45, 15), (120, 59, 37), (128, 64, 32), (200, 99, 53)])
@pytest.mark.parametrize("n", [0, 2])
def test_every_kind_of_host_memory(shape, n):
    import torch
    step, st = _case(*shape)
    ins = [st[k] for k in gu.FIELDS]
    want = step.advance(JaxStateG(*gu.to_device(st), 0.0), n)
    want = [getattr(want, k).cpu().numpy() for k in gu.FIELDS]

    outs = [np.full_like(x, np.nan) for x in ins]
    before = [x.copy() for x in ins]
    _host_step(step, ins, outs, n)
    for name, a, b, x, y in zip(gu.FIELDS, outs, want, ins, before):
        assert np.array_equal(a, b), name
        assert np.array_equal(x, y), name

    # results one float past a page start, with guard values on both sides
    room = [np.full(x.size + 64, 7.0, np.float32) for x in ins]
    odd = [r[17:17 + x.size].reshape(x.shape) for r, x in zip(room, ins)]
    _host_step(step, ins, odd, n)
    for r, a, b in zip(room, odd, want):
        assert np.array_equal(a, b)
        assert (r[:17] == 7.0).all() and (r[17 + a.size:] == 7.0).all()

    pinned = [torch.as_tensor(x).pin_memory() for x in ins]
    _host_step(step, [t.numpy() for t in pinned], outs, n)       # pinned in, pageable out
    assert all(np.array_equal(a, b) for a, b in zip(outs, want))

    _host_step(step, ins, ins, n)                                # in place
    assert all(np.array_equal(a, b) for a, b in zip(ins, want))


@pytest.mark.parametrize("shape", [(180, 90, 19), (200, 99, 53), (360, 180, 25)])
def test_calls_before_and_after_the_slots_are_made(shape):
    """States of 5 and 17 MB: the first calls of a handle copy directly, the
    later ones are staged (from 32 MB in all on); 26 MB are staged at once.
    All give the same results."""
    step, st = _case(*shape)
    ins = [st[k] for k in gu.FIELDS]
    want = step.advance(JaxStateG(*gu.to_device(st), 0.0), 1)
    want = [getattr(want, k).cpu().numpy() for k in gu.FIELDS]
    for _ in range(9):
        outs = [np.full_like(x, np.nan) for x in ins]
        _host_step(step, ins, outs, 1)
        assert all(np.array_equal(a, b) for a, b in zip(outs, want))
