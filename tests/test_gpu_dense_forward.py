"""The tensor-core forward for bf16 storage (densified tiles of 64 outputs): ragged last tiles and panels, batches of one
and several tiles, fan-ins of one and two entries per lane, repeated inputs in a row (few: the list; many: further rounds of
a tile), zero weights, both epilogues."""
import numpy as np
import pytest
import torch

import oracle
from ecml23_sparse_b200 import ops, synth
from cases import ATOL, RTOL, assert_close, config_style_inputs, to_cuda

pytestmark = pytest.mark.gpu


def bf16_case(dev, B, N, L, K, seed, repeats):
    x, idx, W, _ = config_style_inputs(B, N, L, K, seed=seed)
    if repeats == "some":
        idx = synth.indices_with_replacement(seed, 12, L, K, N).numpy()
    elif repeats == "all":
        idx[:, :] = idx[:, :1]           # a row reads one input K times
    W[::7, ::3] = 0.0
    xd, Wd = to_cuda(x, dev).to(torch.bfloat16), to_cuda(W, dev).to(torch.bfloat16)
    return xd, to_cuda(idx, dev), Wd, xd.float().cpu().numpy(), idx, Wd.float().cpu().numpy()


@pytest.mark.parametrize("shape", [(65, 256, 64, 32), (128, 768, 1_001, 32), (100, 320, 130, 40), (256, 512, 777, 64),
                                   (130, 129, 20_003, 16), (70, 128, 37, 16), (97, 700, 300, 31), (128, 768, 130, 64)],
                         ids=lambda s: "B{}_N{}_L{}_K{}".format(*s))
@pytest.mark.parametrize("repeats", ["none", "some", "all"])
def test_dense_forward_matches_the_oracle(cuda_device, shape, repeats):
    dev = cuda_device
    B, N, L, K = shape
    xd, idd, Wd, x, idx, W = bf16_case(dev, B, N, L, K, 31, repeats)
    bias = synth.normal(31, 40, (L,), std=0.5).numpy()
    ref = oracle.forward_f64(x, idx, W, bias=bias)
    for transposed in (False, True):
        xin = xd.t().contiguous() if transposed else xd
        y = ops._forward(xin, idd, Wd, to_cuda(bias, dev), transposed)
        assert_close(y.cpu().numpy(), ref, RTOL, ATOL, "y")
        assert torch.equal(y, ops._forward(xin, idd, Wd, to_cuda(bias, dev), transposed))


@pytest.mark.parametrize("shape", [(65, 384, 64, 32), (128, 768, 1_001, 32), (100, 300, 37, 41), (256, 768, 777, 64)],
                         ids=lambda s: "B{}_N{}_L{}_K{}".format(*s))
@pytest.mark.parametrize("repeats", ["none", "some"])
@pytest.mark.parametrize("loss_name", ["bce", "squared_hinge"])
def test_dense_forward_loss_matches_the_oracle(cuda_device, shape, repeats, loss_name):
    dev = cuda_device
    B, N, L, K = shape
    xd, idd, Wd, x, idx, W = bf16_case(dev, B, N, L, K, 37, repeats)
    bias = synth.normal(37, 40, (L,), std=0.5).numpy()
    row_ptr, labels = synth.multi_hot_targets(37, 41, B, L)
    loss, gT = ops.forward_bce(xd, idd, Wd, to_cuda(bias, dev), row_ptr, labels, False, loss=loss_name)
    z = oracle.forward_f64(x, idx, W, bias=bias).astype(np.float32)
    if loss_name == "bce":
        loss_ref, g_ref = oracle.bce_f64(z, row_ptr.numpy(), labels.numpy())
        assert_close(gT[:, :B].t().cpu().numpy(), g_ref, 5e-5, 2e-7 / (B * L), "gradient")
    else:
        loss_ref, g_ref = oracle.hinge_f64(z, row_ptr.numpy(), labels.numpy(), squared=True)
        assert np.abs(gT[:, :B].t().cpu().numpy() - g_ref).max() <= 4e-5 / (B * L) * max(1.0, np.abs(z).max())
    assert abs(float(loss) - loss_ref) <= 2e-5 * abs(loss_ref) + 1e-7
    assert not gT[:, B:].any()


@pytest.mark.parametrize("shape", [(65, 384, 64, 32), (130, 768, 1_001, 32), (100, 300, 130, 41)],
                         ids=lambda s: "B{}_N{}_L{}_K{}".format(*s))
@pytest.mark.parametrize("repeats", ["none", "some", "all"])
def test_non_finite_inputs_reach_only_the_rows_that_read_them(cuda_device, shape, repeats):
    """Infinities and NaN in single inputs, an all-NaN sample: every logit is what the sum over its row's own entries is."""
    dev = cuda_device
    B, N, L, K = shape
    xd, idd, Wd, clean, idx, W = bf16_case(dev, B, N, L, K, 43, repeats)
    bad = clean.copy()
    bad[3, [0, 6, N - 1]] = np.inf, -np.inf, np.nan
    bad[4, 7] = -np.inf
    bad[B - 1, :] = np.nan
    xd = to_cuda(bad, dev).to(torch.bfloat16)
    bias = synth.normal(43, 40, (L,), std=0.5).numpy()
    with np.errstate(invalid="ignore"):
        ref = np.stack([(W.astype(np.float64) * row[idx]).sum(-1) for row in bad.astype(np.float64)]) + bias
    assert np.isfinite(ref[:B - 1]).any(axis=1).all() and not np.isfinite(ref).all()
    for transposed in (False, True):
        y = ops._forward(xd.t().contiguous() if transposed else xd, idd, Wd, to_cuda(bias, dev), transposed).cpu().numpy()
        finite = np.isfinite(ref)
        assert np.array_equal(np.isnan(y), np.isnan(ref)) and np.array_equal(y[~finite], ref[~finite].astype(np.float32), equal_nan=True)
        assert_close(y[finite], ref[finite], RTOL, ATOL, "y")

    row_ptr, labels = synth.multi_hot_targets(43, 41, B, L)
    _, gT = ops.forward_bce(xd, idd, Wd, to_cuda(bias, dev), row_ptr, labels, False)
    _, g_ref = oracle.bce_f64(np.where(finite, ref, 0.0).astype(np.float32), row_ptr.numpy(), labels.numpy())
    assert_close(gT[:, :B].t().cpu().numpy()[finite], g_ref[finite], 5e-5, 2e-7 / (B * L), "gradient")


def test_waits_that_run_out_end_the_kernel(cuda_device):
    """With a limit below what a tile takes every warp gives up, at its own time, while tiles still need further rounds: the
    launch ends, the event is counted, and the next call is right again."""
    import ctypes
    import time

    import cases
    from ecml23_sparse_b200 import _lib

    dev, lib = cuda_device, _lib.load()
    B, N, L, K = 256, 768, 20_000, 32
    xd, idd, Wd, x, idx, W = bf16_case(dev, B, N, L, K, 47, "all")

    def given_up():
        n = ctypes.c_int(-1)
        _lib.check(lib.ffi_wait_timeouts(ctypes.byref(n)))
        return n.value

    before = given_up()
    _lib.check(lib.ffi_set_wait_limit_ticks(1_000))
    try:
        t0 = time.perf_counter()
        ops._forward(xd, idd, Wd, None, False)
        torch.cuda.synchronize()
        assert time.perf_counter() - t0 < 1.0
    finally:
        _lib.check(lib.ffi_set_wait_limit_ticks(4_000_000_000))
    after = given_up()
    assert after > before
    cases.EXPECTED_WAIT_TIMEOUTS += after - before
    assert_close(ops._forward(xd, idd, Wd, None, False).cpu().numpy(), oracle.forward_f64(x, idx, W), RTOL, ATOL, "y")
    assert given_up() == after
