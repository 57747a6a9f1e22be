"""Fan-ins and bases that leave the rows of W and idx off the 16-byte boundaries, in the kernels that copy rows by the warp:
remainders of four and eight, the last row of an odd table (whose words of W end in mid-word for bf16), short tables that
take narrower batch tiles, inputs that are infinite where no row reads them."""
import numpy as np
import pytest
import torch

import oracle
from ecml23_sparse_b200 import ops, synth
from cases import ATOL, RTOL, assert_close, config_style_inputs, gx_atol, to_cuda

pytestmark = pytest.mark.gpu

SHAPES = [(127, 254, 513, 73), (130, 384, 4_001, 63), (9, 64, 47, 5), (40, 768, 9, 33), (64, 600, 20_001, 6),
          (85, 20_000, 729, 11), (251, 18_000, 301, 33), (300, 17_000, 1_001, 12), (12, 17_000, 33, 1), (16, 17_000, 35, 700)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "B{}_N{}_L{}_K{}".format(*s))
@pytest.mark.parametrize("bf16", [False, True])
def test_odd_fan_in_matches_the_oracle(cuda_device, shape, bf16):
    dev = cuda_device
    B, N, L, K = shape
    x, idx, W, g = config_style_inputs(B, N, L, K, seed=K)
    if bf16:
        x = torch.from_numpy(x).to(torch.bfloat16).float().numpy()
        W = torch.from_numpy(W).to(torch.bfloat16).float().numpy()
    store = torch.bfloat16 if bf16 else torch.float32
    bias = synth.normal(K, 40, (L,), std=0.5).numpy()
    xd, idd, Wd, bd = to_cuda(x.T.copy(), dev).to(store), to_cuda(idx, dev), to_cuda(W, dev).to(store), to_cuda(bias, dev)
    ref = oracle.forward_f64(x, idx, W, bias=bias)
    assert_close(ops._forward(xd, idd, Wd, bd, True).cpu().numpy(), ref, RTOL, ATOL, "y")
    vals, _ = ops.forward_topk(xd, idd, Wd, bd, min(5, L), True)
    assert_close(vals.cpu().numpy(), -np.sort(-ref, axis=1)[:, :min(5, L)], RTOL, ATOL, "top-k")

    row_ptr, labels = synth.multi_hot_targets(3, 41, B, L)
    loss, gT = ops.forward_bce(xd, idd, Wd, bd, row_ptr, labels, True)
    loss_ref, g_ref = oracle.bce_f64(ref.astype(np.float32), row_ptr.numpy(), labels.numpy())
    assert_close(gT[:, :B].t().cpu().numpy(), g_ref, 5e-5, 2e-7 / (B * L), "gradient")
    assert abs(float(loss) - loss_ref) <= 2e-5 * abs(loss_ref) + 1e-7
    assert not gT[:, B:].any()

    gx, gw = ops.fan_in_sparse_matmul_grad_tp(xd, idd, Wd, to_cuda(g, dev))
    assert_close(gw.cpu().numpy(), oracle.grad_w_f64(x, idx, g), RTOL, ATOL, "grad_W")
    assert_close(gx.t().cpu().numpy(), oracle.grad_x_f64(idx, W, g, N), RTOL, gx_atol(L, K, N), "grad_x")


def test_rows_off_the_16_byte_boundaries(cuda_device):
    """K % 4 == 0, but idx and W start one element into their storage; x is infinite where nothing reads it."""
    dev = cuda_device
    for B, N, L, K in ((64, 300, 999, 32), (40, 17_000, 501, 16)):
        x, idx, W, _ = config_style_inputs(B, N, L, K, seed=2)
        idx[idx == 0] = 1
        ref = oracle.forward_f64(x, idx, W)
        x[:, 0] = np.inf
        off = lambda a: torch.cat([a.new_zeros(1), a.reshape(-1)])[1:].view(L, K)
        y = ops._forward(to_cuda(x.T.copy(), dev), off(to_cuda(idx, dev)), off(to_cuda(W, dev)), None, True)
        assert_close(y.cpu().numpy(), ref, RTOL, ATOL, "y")
