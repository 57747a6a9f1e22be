"""One-pass backward (narrow inputs) on tables whose inputs have very different numbers of entries, with infinite and NaN
gradients: the lane groups of a warp walk runs of unequal length, and what a group without an entry reads must not show."""
import pytest
import torch

from ecml23_sparse_b200 import ops

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


@pytest.mark.parametrize("B", [5, 16, 30, 64, 100, 200])
@pytest.mark.parametrize("hot", [1, 12])
@pytest.mark.parametrize("bf16", [False, True])
def test_uneven_runs(B, hot, bf16):
    N, L, K = 700, 6011, 24
    gen = torch.Generator(device="cuda")
    gen.manual_seed(B + hot)
    dt = torch.bfloat16 if bf16 else torch.float32
    x = torch.randn((N, B), generator=gen, device="cuda").to(dt)
    idx = torch.randint(0, N - 100, (L, K), generator=gen, dtype=torch.int32, device="cuda")  # the last 100 have no entry
    idx[:, :3] = idx[:, :3] % hot      # one input with three entries in every row, or twelve with one in every fourth
    W = torch.randn((L, K), generator=gen, device="cuda").to(dt)
    g = torch.randn((L, B), generator=gen, device="cuda")
    g[77, 1], g[5000, B - 1] = float("inf"), float("nan")
    ldg = 32 if B <= 32 else 64 if B <= 64 else (B + 127) // 128 * 128
    gT = torch.zeros((L, ldg), device="cuda")
    gT[:, :B] = g
    plan = ops.FFIPlan(idx, N)
    gx, gw, gb = ops._backward(x, idx, W, gT, True, plan=plan, want_bias_grad=True, grad_is_transposed=True)

    bad_rows = torch.zeros(L, dtype=torch.bool, device="cuda")
    bad_rows[[77, 5000]] = True
    assert not torch.isfinite(gw[bad_rows]).any() and torch.isfinite(gw[~bad_rows]).all()
    assert torch.equal(~torch.isfinite(gb), bad_rows)
    bad = torch.zeros((N, B), dtype=torch.bool, device="cuda")
    bad[idx[77].long(), 1] = True
    bad[idx[5000].long(), B - 1] = True
    assert torch.equal(~torch.isfinite(gx), bad)

    gd, xd, Wd = torch.where(torch.isfinite(g), g, 0.).double(), x.double(), W.double()
    rx, rx_abs = torch.zeros_like(xd), torch.zeros_like(xd)
    rw, rw_abs = torch.empty_like(Wd), torch.empty_like(Wd)
    for k in range(K):
        i = idx[:, k].long()
        t = Wd[:, k, None] * gd
        rx.index_add_(0, i, t)
        rx_abs.index_add_(0, i, t.abs())
        t = xd[i] * gd
        rw[:, k], rw_abs[:, k] = t.sum(1), t.abs().sum(1)
    # a sum of n products in fp32, in any order, is off by at most n * 2^-24 times the sum of magnitudes
    runs = torch.bincount(idx.flatten().long(), minlength=N).double()[:, None] + 8
    assert (((gx.double() - rx).abs() <= runs * EPS * rx_abs + 1e-30) | bad).all()
    assert (((gw.double() - rw).abs() <= (B + 8) * EPS * rw_abs)[~bad_rows]).all()
