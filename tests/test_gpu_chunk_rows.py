"""The one-pass backward over the range of chunk heights and slicings that a plan picks: tables shorter than one chunk per
SM, slices of uneven width, batches of several 128-column tiles (whole, ragged, and with a narrow last tile)."""
import pytest
import torch

import oracle
from ecml23_sparse_b200 import ops
from cases import ATOL, RTOL, assert_close, config_style_inputs, gx_atol, to_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(127, 254, 513, 73), (64, 83, 932, 64), (40, 64, 7, 12), (128, 300, 5_001, 32),
                                   (20, 300, 9_001, 40), (256, 512, 3_001, 64), (129, 151, 2_003, 32), (200, 768, 4_111, 24),
                                   (320, 100, 1_000, 7), (3, 1_000, 40_003, 8)],
                         ids=lambda s: "B{}_N{}_L{}_K{}".format(*s))
@pytest.mark.parametrize("bf16", [False, True])
def test_one_pass_backward_matches_the_oracle(cuda_device, shape, bf16):
    dev = cuda_device
    B, N, L, K = shape
    x, idx, W, g = config_style_inputs(B, N, L, K, seed=23)
    store = torch.bfloat16 if bf16 else torch.float32
    xd, Wd = to_cuda(x, dev).to(store), to_cuda(W, dev).to(store)
    x, W = xd.float().cpu().numpy(), Wd.float().cpu().numpy()
    idd, gd = to_cuda(idx, dev), to_cuda(g, dev)
    gx, gw, gb = ops._backward(xd, idd, Wd, gd, False, want_bias_grad=True)
    assert_close(gw.cpu().numpy(), oracle.grad_w_f64(x, idx, g), RTOL, ATOL * max(1.0, B ** 0.5 / 8), "grad_W")
    assert_close(gx.cpu().numpy(), oracle.grad_x_f64(idx, W, g, N), RTOL, gx_atol(L, K, N), "grad_x")
    gT, _ = ops.transpose_gradient(gd)
    gx2, gw2, gb2 = ops._backward(xd, idd, Wd, gT, False, want_bias_grad=True, grad_is_transposed=True)
    assert torch.equal(gx, gx2) and torch.equal(gw, gw2)
    for b in (gb, gb2):
        assert_close(b.cpu().numpy(), oracle.grad_bias_f64(g), RTOL, ATOL * max(1.0, B ** 0.5 / 4), "grad_bias")
    info = ops.get_plan(idd, N).info()
    assert info["chunk_rows"] % 8 == 0 and 8 <= info["chunk_rows"] <= 512


@pytest.mark.parametrize("shape", [(130, 300, 999, 33), (40, 64, 7, 12), (200, 768, 4_111, 24), (5, 254, 513, 73)],
                         ids=lambda s: "B{}_N{}_L{}_K{}".format(*s))
def test_bf16_weights_off_the_word_boundary(cuda_device, shape):
    """W starts one element into its storage: the 4-byte copies of the one-pass kernel cannot read it."""
    dev = cuda_device
    B, N, L, K = shape
    x, idx, W, g = config_style_inputs(B, N, L, K, seed=29)
    xd, Wd = to_cuda(x, dev).to(torch.bfloat16), to_cuda(W, dev).to(torch.bfloat16)
    off = torch.cat([Wd.new_zeros(1), Wd.reshape(-1)])[1:].view(L, K)
    assert off.data_ptr() % 4 == 2
    idd, gd = to_cuda(idx, dev), to_cuda(g, dev)
    gx, gw, gb = ops._backward(xd, idd, off, gd, False, want_bias_grad=True)
    x, W = xd.float().cpu().numpy(), Wd.float().cpu().numpy()
    assert_close(gw.cpu().numpy(), oracle.grad_w_f64(x, idx, g), RTOL, ATOL * max(1.0, B ** 0.5 / 8), "grad_W")
    assert_close(gx.cpu().numpy(), oracle.grad_x_f64(idx, W, g, N), RTOL, gx_atol(L, K, N), "grad_x")
    assert_close(gb.cpu().numpy(), oracle.grad_bias_f64(g), RTOL, ATOL * max(1.0, B ** 0.5 / 4), "grad_bias")
