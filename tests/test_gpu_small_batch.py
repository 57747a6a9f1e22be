"""The small-batch forward (batch <= 8: lanes along the fan-in) and the top-k selection behind it and behind the batched
kernels, against the CPU oracle: every sample count, fan-ins with idle lanes, ragged last row groups, ties, lists shorter
than k."""
import numpy as np
import pytest
import torch

import oracle
import ecml23_sparse_b200 as ffi
from ecml23_sparse_b200 import ops, synth
from cases import ATOL, RTOL, assert_close, config_style_inputs, to_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 2, 3, 5, 8, 9])
@pytest.mark.parametrize("N,L,K", [(768, 5_003, 32), (100, 33, 4), (300, 1_001, 72), (32_768, 301, 64), (50, 7, 12)])
@pytest.mark.parametrize("bf16", [False, True])
def test_forward_and_topk_of_a_few_samples(cuda_device, B, N, L, K, bf16):
    dev = cuda_device
    x, idx, W, _ = config_style_inputs(B, N, L, K, seed=B)
    if bf16:
        x = torch.from_numpy(x).to(torch.bfloat16).float().numpy()
        W = torch.from_numpy(W).to(torch.bfloat16).float().numpy()
    store = torch.bfloat16 if bf16 else torch.float32
    bias = synth.normal(B, 40, (L,), std=0.5).numpy()
    ref = oracle.forward_f64(x, idx, W, bias=bias)
    args = (to_cuda(idx, dev), to_cuda(W, dev).to(store), to_cuda(bias, dev))
    for transposed in (True, False):
        xin = to_cuda(np.ascontiguousarray(x.T) if transposed else x, dev).to(store)
        assert_close(ops._forward(xin, *args, transposed).cpu().numpy(), ref, RTOL, ATOL, "y")
        vals, lab = ops.forward_topk(xin, *args, 5, transposed, label_offset=3)
        want = -np.sort(-ref, axis=1)[:, :5]
        assert_close(vals.cpu().numpy(), want, RTOL, ATOL, "top-k values")
        assert_close(vals.cpu().numpy(), np.take_along_axis(ref, lab.cpu().numpy().astype(np.int64) - 3, axis=1), RTOL, ATOL,
                     "value of label")


@pytest.mark.parametrize("B,L", [(1, 6_000), (8, 2_049), (40, 100_003), (128, 200_001)])
def test_topk_breaks_ties_by_label(cuda_device, B, L):
    """Few distinct logits: every rank is decided by the lower label, across lists, segments and shared bounds."""
    dev = cuda_device
    N, K = 64, 4
    idx = synth.indices_without_replacement(5, 0, L, K, N).to(dev)
    W = (synth.indices_with_replacement(5, 1, L, K, 2) - 0.5).to(torch.float32).to(dev)
    x = torch.ones((N, B), device=dev)
    vals, lab = ops.forward_topk(x, idx, W, None, 8, True)
    y = ops._forward(x, idx, W, None, True)
    order = torch.sort(y, dim=1, descending=True, stable=True)
    assert torch.equal(lab.long(), order.indices[:, :8]) and torch.equal(vals, order.values[:, :8])


def test_topk_of_fewer_rows_than_k(cuda_device):
    x = torch.ones((16, 2), device=cuda_device)
    idx = torch.arange(12, dtype=torch.int32, device=cuda_device).reshape(3, 4)
    W = torch.tensor([[1.0], [3.0], [2.0]], device=cuda_device).expand(3, 4).contiguous()
    vals, lab = ops.forward_topk(x, idx, W, None, 5, True)
    assert lab.tolist() == [[1, 2, 0, -1, -1]] * 2 and vals[:, :3].tolist() == [[12.0, 8.0, 4.0]] * 2


def test_adam_step_of_several_parameters_matches_one_by_one(cuda_device):
    """One launch for all parameters: sizes with and without a remainder, unaligned views, both storage types, more than
    one group of eight."""
    dev = cuda_device
    sizes = [1, 3, 4, 1_001, 70_001, 8, 2_000_003, 17, 5]
    base = [synth.normal(3, j, (n + 1,)).to(dev) for j, n in enumerate(sizes)]
    def params():
        return [(b[1:].clone() if j % 3 == 0 else b.clone()[1:]).to(torch.bfloat16 if j % 2 else torch.float32)
                for j, b in enumerate(base)]
    grads = [synth.normal(4, j, (n,)).to(dev) for j, n in enumerate(sizes)]
    together = ffi.FusedAdam(params())
    for _ in range(2):
        together.step(grads)
    for j in range(len(sizes)):
        alone = ffi.FusedAdam([params()[j]])
        for _ in range(2):
            alone.step([grads[j]])
        assert torch.equal(alone.params[0], together.params[j])
        assert torch.equal(alone.m[0], together.m[j]) and torch.equal(alone.v[0], together.v[j])
