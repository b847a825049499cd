"""The learned-closure MLP kernels against the float64 CPU oracle
(oracle/mlp.py): tensor-core BF16 inference, float32 gradients of the masked
mean-square loss, and Adam training."""
import numpy as np
import pytest

from oracle import mlp as omlp

pytestmark = pytest.mark.gpu

INFER_TOL = 5e-3     # BF16 operands; accumulation order and GELU rounding differ
GRAD_TOL = 1e-4      # float32 GPU gradients against float64


def _bf16(a):
    import torch
    return torch.as_tensor(np.asarray(a, dtype=np.float32)).to(torch.bfloat16).to(torch.float32).double().numpy()


def _rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("ncol", [128, 1000])
def test_tensor_core_inference_matches_oracle(ncol):
    import torch
    from zhenmode_b200.closure import ClosureMLP, init_params
    p = init_params(seed=3, out_bias=0.5)
    p[:] += np.random.default_rng(4).standard_normal(p.size).astype(np.float32) * 0.01
    net = ClosureMLP(p)
    X = np.random.default_rng(5).standard_normal((ncol, 256)).astype(np.float32)
    X[:, 252:] = 0.0
    got = net.forward_bf16(torch.as_tensor(X, device="cuda")).cpu().numpy()
    net.check_error()
    want = omlp.forward_bf16(p, X, _bf16)
    assert _rel(got, want) < INFER_TOL, _rel(got, want)
    # a second call on the same object gives the same bits
    again = net.forward_bf16(torch.as_tensor(X, device="cuda")).cpu().numpy()
    assert np.array_equal(got, again)


def test_gradients_match_oracle():
    import torch
    from zhenmode_b200.closure import ClosureMLP, init_params
    rng = np.random.default_rng(7)
    p = init_params(seed=8, out_bias=0.0)
    B = 96
    X = rng.standard_normal((B, 256)).astype(np.float32)
    T = rng.standard_normal((B, 64)).astype(np.float32)
    M = (rng.random((B, 64)) < 0.7).astype(np.float32)
    net = ClosureMLP(p)
    loss, g = net.grad(*(torch.as_tensor(a, device="cuda") for a in (X, T, M)))
    want_loss, want_g = omlp.loss_and_grad(p, X, T, M)
    assert abs(loss - want_loss) <= GRAD_TOL * want_loss
    g = g.cpu().numpy()
    for name in omlp.OFF:
        sl = slice(omlp.OFF[name], omlp.OFF[name] + int(np.prod(omlp.SHAPES[name])))
        assert _rel(g[sl], want_g[sl]) < GRAD_TOL, (name, _rel(g[sl], want_g[sl]))


def test_training_reduces_loss():
    """Adam on a smooth synthetic map: the loss falls by more than 10x."""
    import torch
    from zhenmode_b200.closure import ClosureMLP
    rng = np.random.default_rng(11)
    B = 2048
    X = rng.standard_normal((B, 256)).astype(np.float32) * 0.5
    A = rng.standard_normal((256, 64)).astype(np.float32) / 16.0
    T = np.tanh(X @ A).astype(np.float32)
    M = np.ones_like(T)
    net = ClosureMLP(seed=1)
    net.params[-64:] = 0.0
    Xd, Td, Md = (torch.as_tensor(a, device="cuda") for a in (X, T, M))
    first = net.grad(Xd, Td, Md)[0]
    for _ in range(300):
        net.train_step(Xd, Td, Md, lr=2e-3)
    last = net.grad(Xd, Td, Md)[0]
    assert last < first / 10.0, (first, last)


@pytest.mark.parametrize("B", [1, 15, 64, 129, 4095, 4096, 4097])
@pytest.mark.parametrize("offset", [0, 1])
def test_gradients_at_tile_edges(B, offset):
    """Batches around the row tiles, the batch splits and the switch of tile
    size, with rows that start off a 16-byte boundary.  Each gradient is a sum
    of float32 products; its rounding error is bounded by the summed magnitudes
    times 2^-24 per operation of a chain, far below GRAD_TOL of its norm."""
    import torch
    from zhenmode_b200.closure import ClosureMLP, init_params
    rng = np.random.default_rng(B + 31)
    p = init_params(seed=8, out_bias=0.0)
    X = rng.standard_normal((B, 256)).astype(np.float32)
    T = rng.standard_normal((B, 64)).astype(np.float32)
    M = (rng.random((B, 64)) < 0.7).astype(np.float32)
    M[0, 0] = 1.0

    def dev(a):
        flat = torch.zeros(a.size + offset, device="cuda")
        flat[offset:] = torch.as_tensor(a.ravel(), device="cuda")
        return flat[offset:].view(a.shape)

    net = ClosureMLP(p)
    loss, g = net.grad(dev(X), dev(T), dev(M))
    want_loss, want_g = omlp.loss_and_grad(p, X, T, M)
    assert abs(loss - want_loss) <= GRAD_TOL * want_loss
    g = g.cpu().numpy()
    for name in omlp.OFF:
        sl = slice(omlp.OFF[name], omlp.OFF[name] + int(np.prod(omlp.SHAPES[name])))
        assert _rel(g[sl], want_g[sl]) < GRAD_TOL, (name, _rel(g[sl], want_g[sl]))


@pytest.mark.parametrize("ncol", [1, 31, 127, 128, 129, 37889])
@pytest.mark.parametrize("kind", ["float32", "bfloat16", "float64", "offset"])
def test_inference_rows_and_types(ncol, kind):
    """Ragged row counts (one wave of CTAs and a row) and every way the rows may
    come: float32 rows are rounded to BF16 in the kernel, others before it, so
    all give the same bits; against the oracle at the bound above."""
    import torch
    from zhenmode_b200.closure import ClosureMLP, init_params
    p = init_params(seed=3, out_bias=0.5)
    p[:] += np.random.default_rng(4).standard_normal(p.size).astype(np.float32) * 0.01
    net = ClosureMLP(p)
    X = 2.0 * np.random.default_rng(ncol).standard_normal((ncol, 256)).astype(np.float32)
    X[0, :8] = [60.0, -60.0, 0.0, -0.0, 1e-30, -1e-30, 9.0, -9.0]
    Xd = torch.as_tensor(X, device="cuda")
    base = net.forward_bf16(Xd)
    if kind == "offset":
        flat = torch.zeros(X.size + 1, device="cuda")
        flat[1:] = Xd.reshape(-1)
        got = net.forward_bf16(flat[1:].view(ncol, 256))
    else:
        got = net.forward_bf16(Xd.to(getattr(torch, kind)))
    net.check_error()
    assert torch.equal(got, base)
    rows = np.unique(np.concatenate([np.arange(min(ncol, 300)), np.arange(max(0, ncol - 300), ncol)]))
    want = omlp.forward_bf16(p, X[rows], _bf16)
    assert _rel(got.cpu().numpy()[rows], want) < INFER_TOL


@pytest.mark.parametrize("ncol", [100, 37889, 150000])
def test_a_wait_that_runs_out_ends_every_warp(ncol):
    """Half of the epilogue warps give up in the first pass: the kernel ends (one
    pass a CTA, a second one in one CTA, several in all), sets its error word, and
    the next inference is right."""
    import ctypes
    import torch
    from zhenmode_b200.closure import ClosureMLP
    net = ClosureMLP(seed=2)
    X = torch.randn((ncol, 256), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").bfloat16()
    want = net.forward_bf16(X)
    net.check_error()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    Y = torch.empty((ncol, 64), device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert net.lib.zm_mlp_wait_probe(stream, ncol, p(X), p(net.Wp), p(net.b1), p(net.b2), p(net.b3), p(Y),
                                     p(net.err)) == 0
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError):
        net.check_error()
    net.err.zero_()
    assert torch.equal(net.forward_bf16(X), want)
    net.check_error()


def test_gelu_of_the_inference_on_both_sides():
    """One feature through one unit of each hidden layer, scaled between them by
    2^23, where GELU is the identity (exactly, in BF16) or vanishes: output 0 is
    |gelu(x)| for negative x, output 1 gelu(x) for positive.  The hidden value is
    rounded to BF16 once and the rest is exact, so the outputs are BF16 numbers:
    the one nearest to the float64 value, or its neighbour where the kernel's GELU
    (well below a step of 2^-8 off) falls to the other side of a rounding boundary."""
    import math
    import torch
    from zhenmode_b200.closure import N_PARAMS, ClosureMLP, unpack
    p = np.zeros(N_PARAMS, np.float32)
    w = unpack(p)
    s = 2.0 ** 23
    w["W1"][0, 0] = 1.0
    w["W2"][0, 0], w["W2"][1, 0] = -s, s
    w["W3"][0, 0] = w["W3"][1, 1] = 1.0 / s
    net = ClosureMLP(p)
    x = torch.cat([-torch.linspace(2.0 ** -7, 5.0, 4000), torch.linspace(2.0 ** -7, 60.0, 4000)]).bfloat16()
    X = torch.zeros((x.numel(), 256), dtype=torch.bfloat16)
    X[:, 0] = x
    y = net.forward_bf16(X.cuda()).double().cpu().numpy()
    net.check_error()
    x = x.double().numpy()
    want = x * np.array([0.5 * math.erfc(-v / math.sqrt(2.0)) for v in x])
    got = np.where(x < 0, -y[:, 0], y[:, 1])
    step = torch.as_tensor(want).bfloat16().view(torch.int16).int() - torch.as_tensor(got).bfloat16().view(torch.int16).int()
    assert np.array_equal(torch.as_tensor(got).bfloat16().double().numpy(), got)
    assert int(step.abs().max()) <= 1
    assert np.max(np.abs(np.where(x < 0, y[:, 1], y[:, 0]))) < 1e-30  # |gelu(z)| <= 12 Phi(-12) = 2e-32


def test_rows_with_nan_and_infinities_stay_alone():
    """Non-finite features make their own row NaN (a hidden value of -inf has none) and no other."""
    import torch
    from zhenmode_b200.closure import ClosureMLP
    net = ClosureMLP(seed=2)
    X = torch.randn((300, 256), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    want = net.forward_bf16(X)
    bad = X.clone()
    bad[5, 3], bad[130, 7], bad[299, 0] = float("nan"), float("inf"), float("-inf")
    got = net.forward_bf16(bad)
    net.check_error()
    rows = torch.ones(300, dtype=torch.bool, device="cuda")
    rows[[5, 130, 299]] = False
    assert torch.equal(got[rows], want[rows])
    assert got[~rows].isnan().all()


def _ptr(t):
    import ctypes
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("ncol", [0, 1, 129, 37889, 80000])
def test_weights_in_rows_give_the_packed_ones_bits(ncol):
    """The same chunks of the same BF16 weights, fetched from their rows: the same products in the same order."""
    import ctypes
    import torch
    from zhenmode_b200.closure import ClosureMLP
    net = ClosureMLP(seed=4)
    X = torch.randn((max(ncol, 1), 256), generator=torch.Generator(device="cuda").manual_seed(ncol), device="cuda")
    X = X.bfloat16()
    want = net.forward_bf16(X)
    W = [torch.empty(s, dtype=torch.bfloat16, device="cuda") for s in ((256, 256), (256, 256), (64, 256))]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert net.lib.zm_mlp_pack_bf16(stream, _ptr(net.params), *[_ptr(w) for w in W]) == 0
    Y = torch.full((max(ncol, 1), 64), 7.0, device="cuda")

    def call(x, w1):
        return net.lib.zm_mlp_forward_bf16(stream, ncol, x, w1, _ptr(net.b1), _ptr(W[1]), _ptr(net.b2), _ptr(W[2]),
                                           _ptr(net.b3), _ptr(Y), _ptr(net.err))

    assert call(_ptr(X), _ptr(W[0])) == 0
    net.check_error()
    assert torch.equal(Y, want) if ncol else bool((Y == 7.0).all())
    off = ctypes.c_void_p(W[0].data_ptr() + 2)  # rows off a 16-byte boundary are refused
    assert call(_ptr(X), off) != 0 and call(ctypes.c_void_p(X.data_ptr() + 2), _ptr(W[0])) != 0


def test_the_weights_of_a_network_may_be_replaced():
    """W1, W2, W3 hold the BF16 weights of the last pack(); written in place or
    set, the inference follows them, and pack() returns to the parameters."""
    import torch
    from zhenmode_b200.closure import ClosureMLP, unpack
    net, other = ClosureMLP(seed=4), ClosureMLP(seed=9)
    X = torch.randn((500, 256), device="cuda")
    mine, theirs = net.forward_bf16(X), other.forward_bf16(X)
    for a, b in zip((net.W1, net.W2, net.W3), ("W1", "W2", "W3")):
        assert torch.equal(a, unpack(net.params)[b].bfloat16())
    assert torch.equal(net.forward_bf16(X), mine)
    net.W1 = other.W1.clone()
    net.W2.copy_(other.W2)
    net.W3 = other.W3
    net.b3.copy_(other.b3)
    assert torch.equal(net.forward_bf16(X), theirs)
    net.params.mul_(1.0)
    net.pack()
    net.b3 = unpack(ClosureMLP(seed=4).params)["b3"].contiguous()
    assert torch.equal(net.forward_bf16(X), mine)
    # weights read before the parameters change are those of the last pack()
    later = ClosureMLP(seed=4)
    later.params.zero_()
    assert torch.equal(later.W2, unpack(ClosureMLP(seed=4).params)["W2"].bfloat16())
