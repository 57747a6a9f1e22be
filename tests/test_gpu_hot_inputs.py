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


@pytest.mark.parametrize("B", [7, 16, 17, 64, 128, 150])
@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("shares", [
    ((0, 0.2),),                                  # one hot input, first of its warp
    ((31, 0.35), (30, 0.05)),                     # two of a warp and bundle, unequal
    ((100, 0.05), (101, 0.05), (102, 0.05), (103, 0.05)),  # a bundle that is even in itself
    ((299, 0.6),),                                # the last input
    ((8, 0.02), (40, 0.02), (77, 0.01), (111, 0.005)),     # around the length from which on a run is shared
    ((5, 1.0),),                                  # nothing else: no chunk has another input
])
def test_hot_inputs(B, bf16, shares):
    """What a run has more than the others of its bundle is walked by all lane groups: remainders of all kinds."""
    _check_shares(300, B, bf16, shares)


@pytest.mark.parametrize("B", [7, 16, 17, 64, 128, 150])
@pytest.mark.parametrize("shares", [((31, 0.35), (30, 0.05)), ((249, 0.6),), ((5, 1.0),)])
def test_hot_inputs_of_one_slice(B, shares):
    """With more than one slice the hottest of these tables go to a kernel for each gradient."""
    _check_shares(250, B, B % 2 == 0, shares)


def _check_shares(N, B, bf16, shares):
    L, K = 9001, 24
    gen, x, W, g = _inputs(B, N, L, K, torch.bfloat16 if bf16 else torch.float32, B)
    idx = torch.randint(0, N, (L, K), generator=gen, dtype=torch.int32, device="cuda")
    u = torch.rand((L, K), generator=gen, device="cuda")
    for i, share in shares:
        idx[(u >= 0) & (u < share)] = i
        u -= share
    _check(x, idx, W, g)


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


@pytest.mark.parametrize("B", [16, 32])
def test_hot_inputs_do_not_serialise(B):
    """Inputs drawn by Zipf's law (the first has a seventh of all entries): 3 to 4 times the time of a uniform table where a lane
    group walked such a run by itself 11 to 18 times."""
    N, L, K = 768, 200000, 32
    gen, x, W, g = _inputs(B, N, L, K, torch.float32, B)
    uniform = torch.randint(0, N, (L, K), generator=gen, dtype=torch.int32, device="cuda")
    cdf = torch.cumsum(1.0 / torch.arange(1, N + 1, dtype=torch.float64, device="cuda"), 0)
    u = torch.rand((L, K), generator=gen, dtype=torch.float64, device="cuda") * cdf[-1]
    zipf = torch.randperm(N, generator=gen, device="cuda")[torch.searchsorted(cdf, u).clamp(max=N - 1)].int()
    gT = torch.zeros((L, _stride(B)), device="cuda")
    gT[:, :B] = g
    times = []
    for idx in (uniform, zipf):
        plan = ops.FFIPlan(idx, N)
        times.append(_time(lambda: ops._backward(x, idx, W, gT, True, plan=plan, grad_is_transposed=True)))
    assert times[1] < 8 * times[0]


@pytest.mark.parametrize("N,L,K,B,share", [(2048, 150000, 32, 64, 0.2), (2048, 150000, 32, 32, 0.4), (2048, 150000, 32, 8, 0.8),
                                           (768, 200000, 32, 32, 0.8), (768, 200000, 32, 64, 0.4), (300, 100000, 32, 64, 0.8)])
def test_very_hot_input_is_no_slower_than_two_kernels(N, L, K, B, share):
    """One input with a large part of the links: 1.2 to 3 times the two gradients by themselves in the one-pass kernel."""
    gen, x, W, g = _inputs(B, N, L, K, torch.float32, B)
    idx = torch.randint(0, N, (L, K), generator=gen, dtype=torch.int32, device="cuda")
    idx[torch.rand((L, K), generator=gen, device="cuda") < share] = 17
    gT = torch.zeros((L, _stride(B)), device="cuda")
    gT[:, :B] = g
    plan = ops.FFIPlan(idx, N)

    def time(**want):
        return min(_time(lambda: ops._backward(x, idx, W, gT, True, plan=plan, grad_is_transposed=True, **want)) for _ in range(3))

    assert time() < 1.08 * (time(want_weight_grad=False) + time(want_feature_grad=False))


@pytest.mark.parametrize("B", [1, 9, 24, 64, 127, 200])
@pytest.mark.parametrize("N,L,K,bf16", [(1, 5003, 3, False), (3, 9001, 2, True), (10, 20011, 8, False), (16, 4099, 7, True), (17, 4099, 16, False),
                                        (33, 30001, 5, True), (48, 7001, 24, False), (49, 7001, 24, True), (65, 3001, 16, False),
                                        (32, 9001, 40, True), (48, 40001, 40, False), (100, 500, 72, False)])
def test_few_inputs(B, N, L, K, bf16):
    """Fewer inputs per warp than lane groups, down to warps without any: the groups share the runs where these are long."""
    gen, x, W, g = _inputs(B, N, L, K, torch.bfloat16 if bf16 else torch.float32, B)
    _check(x, torch.randint(0, N, (L, K), generator=gen, dtype=torch.int32, device="cuda"), W, g)


@pytest.mark.parametrize("B", [8, 64, 128])
def test_few_inputs_do_not_idle_the_lane_groups(B):
    """As many entries among 10 inputs as among 256: 1 to 1.2 times the time; 2 to 3 times when a group walked an input by itself."""
    L, K = 300000, 8
    times = []
    for N in (256, 10):
        gen, x, W, g = _inputs(B, N, L, K, torch.float32, B)
        idx = torch.randint(0, N, (L, K), generator=gen, dtype=torch.int32, device="cuda")
        gT = torch.zeros((L, _stride(B)), device="cuda")
        gT[:, :B] = g
        plan = ops.FFIPlan(idx, N)
        times.append(min(_time(lambda: ops._backward(x, idx, W, gT, True, plan=plan, grad_is_transposed=True)) for _ in range(3)))
    assert times[1] < 1.6 * times[0]


def _weighted_table(weights, L, K, gen):
    cdf = torch.cumsum(weights.double(), 0)
    u = torch.rand((L, K), generator=gen, dtype=torch.float64, device="cuda") * cdf[-1]
    return torch.searchsorted(cdf, u).clamp(max=len(weights) - 1).int()


def _weights(kind, N, gen):
    ranks = torch.arange(1, N + 1, device="cuda")
    if kind == "uniform":
        return torch.ones(N, device="cuda")
    if kind == "leading quarter":  # 30 % of the links more
        w = torch.ones(N, device="cuda")
        w[:N // 4] += 0.3 / 0.7 * 4
        return w
    exponent, order = kind
    w = ranks.double() ** -exponent
    return w if order == "ordered" else w[torch.randperm(N, generator=gen, device="cuda")]


def _kernels(f):
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        for _ in range(3):  # (the profiler may miss single short kernels)
            f()
            torch.cuda.synchronize()
    return [e.name for e in prof.events()]


@pytest.mark.parametrize("kind", [(0.6, "shuffled"), (1.0, "shuffled"), (0.5, "ordered"), "leading quarter", "uniform"], ids=str)
def test_uneven_tables_take_the_one_pass_kernel(kind):
    N, L, K = 768, 670091, 32
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    idx = _weighted_table(_weights(kind, N, gen), L, K, gen)
    W = torch.randn((L, K), generator=gen, device="cuda")
    plan = ops.FFIPlan(idx, N)
    for B in (16, 64, 128):
        x, gT = torch.randn((N, B), generator=gen, device="cuda"), torch.zeros((L, _stride(B)), device="cuda")
        names = _kernels(lambda: ops._backward(x, idx, W, gT, True, plan=plan, grad_is_transposed=True))
        assert any("ffi_bwd_runs_kernel" in n for n in names), names
        assert not any("grad_x_narrow" in n for n in names), names


@pytest.mark.parametrize("N,L,K", [(768, 20011, 32), (100, 3001, 7), (15, 900, 3), (513, 40000, 24), (2048, 9000, 16), (300, 33, 5)])
@pytest.mark.parametrize("kind", [(0.8, "shuffled"), (1.2, "ordered"), "leading quarter"], ids=str)
def test_dealt_plans(N, L, K, kind):
    """Plans of uneven tables hold their inputs in another order, and shorter chunks where need be: the index they hold, all entry
    points that read it, and rebuilds from even to uneven tables and back."""
    gen, x, W, g = _inputs(70, N, L, K, torch.float32, 3)
    idx = _weighted_table(_weights(kind, N, gen), L, K, gen)
    even = torch.randint(0, N, (L, K), generator=gen, dtype=torch.int32, device="cuda")
    _check(x, idx, W, g)
    plan = ops.FFIPlan(idx, N)
    for a, b in zip(plan.export(), plan.export(chunked=True)):
        assert torch.equal(a, b)
    gT = torch.zeros((L, 128), device="cuda")
    gT[:, :70] = g

    def grads(plan, idx):
        both = ops._backward(x, idx, W, gT, True, plan=plan, grad_is_transposed=True)
        alone = ops._backward(x, idx, W, gT, True, plan=plan, want_weight_grad=False, grad_is_transposed=True)
        return both[0], both[1], alone[0]

    want, want_even = grads(plan, idx), grads(ops.FFIPlan(even, N), even)
    n = torch.bincount(idx.flatten().long(), minlength=N).double()[:, None] + 8
    size = torch.zeros((N, 70), dtype=torch.float64, device="cuda")
    for k in range(K):
        size.index_add_(0, idx[:, k].long(), (W[:, k, None] * g).abs().double())
    assert ((want[0].double() - want[2].double()).abs() <= 2 * n * EPS * size + 1e-30).all()
    plan.rebuild(even)
    held = plan.info()["device_bytes"]
    for table, values in ((even, want_even), (idx, want), (even, want_even)):
        plan.rebuild(table)
        assert plan.info()["device_bytes"] == held
        for a, b in zip(grads(plan, table), values):
            assert torch.equal(a, b)
        for a, b in zip(plan.export(), plan.export(chunked=True)):
            assert torch.equal(a, b)


@pytest.mark.parametrize("N,L,K", [(254, 513, 73), (64, 1000, 16), (700, 2000, 40)])
def test_plans_of_short_tables_hold_one_set_of_chunks(N, L, K):
    """Their chunks never get shorter, so nothing is kept in hand for that: plan creation grows by jumps with what it allocates."""
    idx = torch.randint(0, N, (L, K), dtype=torch.int32, device="cuda")
    info = ops.FFIPlan(idx, N).info()
    arrays = [(N + 1) * 4, L * K * 4, L * K * 4, info["n_chunks"] * (N + 1) * 4, N * 4]
    assert info["device_bytes"] <= sum((b + 255) // 256 * 256 for b in arrays)
