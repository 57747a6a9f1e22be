"""One-pass backward for wide inputs (csrc/backward_wide.cu) against fp64 sums: edges of its tiles, batches and chunks."""
import pytest
import torch

from ecml23_sparse_b200 import ops

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24

# B, N, L, K, storage, x given as [N,B]
SHAPES = [
    (1, 2049, 70, 3, "f32", True),             # one column, runs of a handful of entries
    (33, 3001, 517, 33, "f32", False),         # odd batch: tile of 64 columns, ragged rows of x, x given as [B,N]
    (64, 20000, 31, 8, "bf16", True),          # most inputs have no entry
    (85, 2500, 4099, 36, "bf16", False),
    (128, 16384, 2000, 32, "f32", True),
    (130, 4096, 1500, 63, "f32", True),        # 256 columns allocated, the second half nearly empty
    (300, 2200, 900, 17, "bf16", True),        # three tiles of 128 columns
    (32, 2111, 400000, 4, "f32", True),        # two chunks of one narrow tile
    (256, 3000, 50021, 8, "bf16", True),       # two chunks of one tile of 256 columns
    (512, 3000, 50021, 5, "f32", False),       # two chunks of two tiles each
    (33, 2111, 250007, 4, "f32", True),        # two chunks, rows of grad_x that are neither aligned nor whole
    (130, 4737, 50021, 5, "bf16", False),      # the same with 256 columns, most of them padding; one input more than resident warps
    (300, 2369, 100003, 4, "f32", True),       # two chunks of three tiles, the last one ragged
]


def _inputs(B, N, L, K, storage, seed=3, hot=True):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    dt = torch.bfloat16 if storage == "bf16" else torch.float32
    x = torch.randn((B, N), generator=gen, device="cuda").to(dt)
    idx = torch.randint(0, N, (L, K), generator=gen, dtype=torch.int32, device="cuda")
    if hot:
        idx[:, 0] = idx[:, 0] % 5      # long runs: several batches of 32 entries per chunk
    W = torch.randn((L, K), generator=gen, device="cuda").to(dt)
    g = torch.randn((B, L), generator=gen, device="cuda")
    return x, idx, W, g


def _reference(x, idx, W, g):
    """fp64 values and the sums of magnitudes that bound the rounding of any order of fp32 additions."""
    xT, gT, W = x.double().t().contiguous(), g.double().t().contiguous(), W.double()
    gx, gx_abs = torch.zeros_like(xT), torch.zeros_like(xT)
    gw, gw_abs = torch.empty_like(W), torch.empty_like(W)
    for k in range(idx.shape[1]):
        i = idx[:, k].long()
        t = W[:, k, None] * gT
        gx.index_add_(0, i, t)
        gx_abs.index_add_(0, i, t.abs())
        t = xT[i] * gT
        gw[:, k], gw_abs[:, k] = t.sum(1), t.abs().sum(1)
    return gx, gx_abs, gw, gw_abs, gT.sum(1), gT.abs().sum(1)


@pytest.mark.parametrize("B,N,L,K,storage,tp", SHAPES)
def test_matches_fp64(B, N, L, K, storage, tp):
    _check(B, N, L, K, storage, tp, True)


@pytest.mark.parametrize("B,N,L,K,storage,tp", [s for s in SHAPES if s[0] > 256])
def test_matches_fp64_without_hot_inputs(B, N, L, K, storage, tp):
    """Several batch tiles: with the hot inputs of the other test such tables go to a kernel for each gradient."""
    _check(B, N, L, K, storage, tp, False)


@pytest.mark.parametrize("B,N,L,K,storage", [(512, 3000, 50021, 5, "f32"), (300, 2369, 100003, 4, "f32"), (256, 3000, 50021, 8, "bf16")])
def test_takes_the_one_pass_kernel(B, N, L, K, storage):
    x, idx, W, g = _inputs(B, N, L, K, storage, hot=B <= 256)
    plan = ops.FFIPlan(idx, N)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        for _ in range(5):  # (the profiler may miss single short kernels)
            ops._backward(x, idx, W, g, False, plan=plan)
            torch.cuda.synchronize()
    names = [e.name for e in prof.events()]
    assert any("ffi_bwd_wide_kernel" in n for n in names), names


def _check(B, N, L, K, storage, tp, hot):
    x, idx, W, g = _inputs(B, N, L, K, storage, hot=hot)
    gx, gx_abs, gw, gw_abs, gb, gb_abs = _reference(x, idx, W, g)
    ldg = 32 if B <= 32 else 64 if B <= 64 else (B + 127) // 128 * 128
    gT = torch.zeros((L, ldg), device="cuda")
    gT[:, :B] = g.t()
    xs = x.t().contiguous() if tp else x
    plan = ops.FFIPlan(idx, N)
    # a sum of n products in fp32, in any order, is off by at most n * 2^-24 times the sum of magnitudes
    runs = torch.bincount(idx.flatten().long(), minlength=N).double()[:, None] + 8
    for from_transposed in (True, False):
        def call():
            return ops._backward(xs, idx, W, gT if from_transposed else g, tp, plan=plan, want_bias_grad=True,
                                 grad_is_transposed=from_transposed)
        ox, ow, ob = call()
        oxT = (ox if tp else ox.t()).double()
        assert ((oxT - gx).abs() <= runs * EPS * gx_abs + 1e-30).all()
        assert ((ow.double() - gw).abs() <= (B + 8) * EPS * gw_abs).all()
        assert ((ob.double() - gb).abs() <= (B + 8) * EPS * gb_abs).all()
        for a, b in zip((ox, ow, ob), call()):
            assert torch.equal(a, b)


def test_captured_and_with_special_values():
    B, N, L, K = 256, 3000, 50021, 8
    x, idx, W, g = _inputs(B, N, L, K, "f32")
    g[7, 49999] = float("nan")
    g[9, 3] = float("inf")
    xs, gT = x.t().contiguous(), g.t().contiguous()
    plan = ops.FFIPlan(idx, N)

    def call():
        return ops._backward(xs, idx, W, gT, True, plan=plan, want_bias_grad=True, grad_is_transposed=True)

    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        want = call()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = call()
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    bad_rows = torch.zeros(L, dtype=torch.bool, device="cuda")
    bad_rows[[49999, 3]] = True
    assert not torch.isfinite(want[1][bad_rows]).any() and torch.isfinite(want[1][~bad_rows]).all()
    bad = torch.zeros((N, B), dtype=torch.bool, device="cuda")
    bad[idx[49999].long(), 7] = True
    bad[idx[3].long(), 9] = True
    assert torch.equal(~torch.isfinite(want[0]), bad)


def _time(f):
    for _ in range(3):
        f()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    for _ in range(5):
        f()
    b.record()
    b.synchronize()
    return a.elapsed_time(b)


@pytest.mark.parametrize("B,N,storage", [(300, 2049, "f32"), (512, 2049, "f32"), (390, 5000, "bf16"), (128, 5000, "f32")])
def test_one_pass_is_no_slower_than_two(B, N, storage):
    """Just above the narrow inputs and a multiple of the resident warps, with several batch tiles: measured 1.1 to 1.4 times as
    fast as the two gradients by themselves, 0.7 to 1.2 when later tiles loaded grad_W and SMs had unequal shares."""
    x, idx, W, g = _inputs(B, N, 200000, 32, storage)
    idx[:, 0] = idx[:, 1].flip(0)     # (no hot inputs)
    xs, gT = x.t().contiguous(), torch.zeros((200000, (B + 127) // 128 * 128), device="cuda")
    gT[:, :B] = g.t()
    _compare_with_two(xs, idx, W, gT, 1.1)


@pytest.mark.parametrize("B,N,L,storage", [(512, 16384, 50000, "bf16"), (640, 5000, 100000, "bf16"), (1024, 32768, 60000, "f32")])
@pytest.mark.parametrize("share", [0.001, 0.01])
def test_hot_inputs_do_not_wait_tile_by_tile(B, N, L, storage, share):
    """An input with many of the links is one warp's work in every batch tile, and the tiles of the one-pass kernel come one after
    another: 1.1 to 1.9 times the two gradients by themselves, which walk all tiles at once, until such tables went to these."""
    x, idx, W, g = _inputs(B, N, L, 32, storage, hot=False)
    idx[torch.rand((L, 32), device="cuda") < share] = 17
    xs, gT = x.t().contiguous(), torch.zeros((L, (B + 127) // 128 * 128), device="cuda")
    gT[:, :B] = g.t()
    _compare_with_two(xs, idx, W, gT, 1.04)


def _compare_with_two(xs, idx, W, gT, most):
    plan = ops.FFIPlan(idx, xs.shape[0])

    def call(**want):
        return ops._backward(xs, idx, W, gT, True, plan=plan, grad_is_transposed=True, **want)

    def time(**want):
        return min(_time(lambda: call(**want)) for _ in range(3))

    assert time() < most * (time(want_weight_grad=False) + time(want_feature_grad=False))
