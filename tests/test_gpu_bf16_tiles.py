"""The bf16 forward in batch tiles of 32, 64 and 128 columns: ragged batches over one and several tiles, short and odd tables, inputs
too wide for the wider tiles, a W that does not start on a 16-byte boundary."""
import numpy as np
import pytest
import torch

import oracle
from ecml23_sparse_b200 import ops, synth
from cases import ATOL, RTOL, assert_close, config_style_inputs, to_cuda

pytestmark = pytest.mark.gpu

SHAPES = [(16, 80, 3_001, 72), (9, 2_900, 501, 8), (32, 768, 5, 72), (59, 455, 2_973, 72), (64, 1_500, 777, 16), (33, 96, 40_001, 80),
          (128, 768, 1_001, 72), (130, 384, 515, 16), (203, 384, 7_210, 16), (500, 80, 1_111, 72), (97, 1_100, 333, 24),
          (130, 384, 515, 64)]  # the last: gathers where the rows start on 16 bytes, the tensor cores where not


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "B{}_N{}_L{}_K{}".format(*s))
@pytest.mark.parametrize("aligned", [True, False])
def test_bf16_forward_tiles_match_the_oracle(cuda_device, shape, aligned):
    dev = cuda_device
    B, N, L, K = shape
    x, idx, W, _ = config_style_inputs(B, N, L, K, seed=B)
    xd, Wd = to_cuda(x.T.copy(), dev).to(torch.bfloat16), to_cuda(W, dev).to(torch.bfloat16)
    if not aligned:
        Wd = torch.cat([Wd.new_zeros(1), Wd.reshape(-1)])[1:].view(L, K)
    bias = synth.normal(B, 40, (L,), std=0.5).numpy()
    idd, bd = to_cuda(idx, dev), to_cuda(bias, dev)
    ref = oracle.forward_f64(xd.float().cpu().numpy().T.copy(), idx, Wd.float().cpu().numpy(), bias=bias)
    assert_close(ops._forward(xd, idd, Wd, bd, True).cpu().numpy(), ref, RTOL, ATOL, "y")
    row_ptr, labels = synth.multi_hot_targets(3, 41, B, L)
    loss, gT = ops.forward_bce(xd, idd, Wd, bd, row_ptr, labels, True)
    loss_ref, g_ref = oracle.bce_f64(ref.astype(np.float32), row_ptr.numpy(), labels.numpy())
    assert_close(gT[:, :B].t().cpu().numpy(), g_ref, 5e-5, 2e-7 / (B * L), "gradient")
    assert abs(float(loss) - loss_ref) <= 2e-5 * abs(loss_ref) + 1e-7
    assert not gT[:, B:].any()
