"""The one-pass backward with 4, 8 and 16 entries per warp step (batch tiles of 32, 16 and 8 columns): batches on both sides of
the limits, narrow last tiles, odd numbers of inputs, runs shorter than a step, wide and narrow chunks."""
import pytest
import torch

import oracle
from ecml23_sparse_b200 import ops
from cases import ATOL, RTOL, assert_close, config_style_inputs, gx_atol, to_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 7, 8, 9, 16, 17, 133, 140])
@pytest.mark.parametrize("N,L,K", [(205, 7_001, 48), (768, 30_011, 32), (67, 40, 5), (1_000, 3_003, 8), (33, 20_001, 24)])
@pytest.mark.parametrize("bf16", [False, True])
def test_one_pass_backward_of_few_columns(cuda_device, B, N, L, K, bf16):
    dev = cuda_device
    x, idx, W, g = config_style_inputs(B, N, L, K, seed=B)
    store = torch.bfloat16 if bf16 else torch.float32
    xd, Wd = to_cuda(x.T.copy(), dev).to(store), to_cuda(W, dev).to(store)
    x, W = xd.float().cpu().numpy().T.copy(), Wd.float().cpu().numpy()
    idd, gd = to_cuda(idx, dev), to_cuda(g, dev)
    gT, _ = ops.transpose_gradient(gd)
    gx, gw, gb = ops._backward(xd, idd, Wd, gT, True, want_bias_grad=True, grad_is_transposed=True)
    assert_close(gw.cpu().numpy(), oracle.grad_w_f64(x, idx, g), RTOL, ATOL * max(1.0, B ** 0.5 / 8), "grad_W")
    assert_close(gx.t().cpu().numpy(), oracle.grad_x_f64(idx, W, g, N), RTOL, gx_atol(L, K, N), "grad_x")
    assert_close(gb.cpu().numpy(), oracle.grad_bias_f64(g), RTOL, ATOL * max(1.0, B ** 0.5 / 4), "grad_bias")
    again = ops._backward(xd, idd, Wd, gd, True)
    assert torch.equal(gx, again[0]) and torch.equal(gw, again[1])
