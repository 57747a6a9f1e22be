"""One-pass backward (narrow inputs) on tables with a few inputs that have a large part of all entries."""
import pytest
import torch

from ecml23_sparse_b200 import ops

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def _stride(B):
    return 32 if B <= 32 else 64 if B <= 64 else (B + 127) // 128 * 128


def _backward(x, idx, W, g, plan):
    gT = torch.zeros((g.shape[0], _stride(g.shape[1])), device="cuda")
    gT[:, :g.shape[1]] = g
    return ops._backward(x, idx, W, gT, True, plan=plan, want_bias_grad=True, grad_is_transposed=True)


def _check(x, idx, W, g):
    N, B = x.shape
    plan = ops.FFIPlan(idx, N)
    gx, gw, gb = _backward(x, idx, W, g, plan)
    gd, xd, Wd = g.double(), x.double(), W.double()
    rx, rx_abs = torch.zeros_like(xd), torch.zeros_like(xd)
    rw, rw_abs = torch.empty_like(Wd), torch.empty_like(Wd)
    for k in range(idx.shape[1]):
        i = idx[:, k].long()
        t = Wd[:, k, None] * gd
        rx.index_add_(0, i, t)
        rx_abs.index_add_(0, i, t.abs())
        t = xd[i] * gd
        rw[:, k], rw_abs[:, k] = t.sum(1), t.abs().sum(1)
    # a sum of n products in fp32, in any order, is off by at most n * 2^-24 times the sum of magnitudes
    runs = torch.bincount(idx.flatten().long(), minlength=N).double()[:, None] + 8
    assert ((gx.double() - rx).abs() <= runs * EPS * rx_abs + 1e-30).all()
    assert ((gw.double() - rw).abs() <= (B + 8) * EPS * rw_abs).all()
    assert ((gb.double() - gd.sum(1)).abs() <= (B + 8) * EPS * gd.abs().sum(1)).all()
    for a, b in zip((gx, gw, gb), _backward(x, idx, W, g, plan)):
        assert torch.equal(a, b)


def _inputs(B, N, L, K, dt, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    x = torch.randn((N, B), generator=gen, device="cuda").to(dt)
    W = torch.randn((L, K), generator=gen, device="cuda").to(dt)
    g = torch.randn((L, B), generator=gen, device="cuda")
    return gen, x, W, g


@pytest.mark.parametrize("B", [3, 8, 16, 32, 64, 128])
@pytest.mark.parametrize("hot", [240, 252, 255])
def test_hot_input_of_the_last_warp(B, hot):
    """Half of all entries belong to one input of a slice's last warp, whose entries end the staging buffer: 3,000 and more a
    chunk, of 8 bytes each, so that a group which reads on at its own run's end while the hot run lasts would leave the shared
    memory behind the buffer (23 KB with 4 groups, 14 with 8, 9 with 16)."""
    N, L, K = 256, 30000, 32
    gen, x, W, g = _inputs(B, N, L, K, torch.float32, B)
    idx = torch.randint(0, N, (L, K), generator=gen, dtype=torch.int32, device="cuda")
    idx[:, ::2] = hot
    _check(x, idx, W, g)
