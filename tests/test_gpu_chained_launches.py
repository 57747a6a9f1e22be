"""Kernels that are set up while the one before them still runs: passes on changing inputs, back to back and out of a CUDA graph, give
what they give one at a time (a kernel that read before its predecessor was done would see the pass before)."""
import pytest
import torch

from ecml23_sparse_b200 import ops

pytestmark = pytest.mark.gpu

# B, N, L, K, storage, x given as [N,B]; small ones, whose kernels are shorter than a launch, and one with long kernels; the last three take the
# one-pass backward for wide inputs, whose launches set each other up and read gT before they wait, in two chunks of one and of two
# batch tiles
SHAPES = [(127, 254, 513, 73, "f32", False), (5, 64, 40, 8, "f32", True), (20, 205, 900, 16, "bf16", True), (130, 300, 2000, 24, "bf16", False),
          (33, 3000, 700, 8, "f32", False), (128, 768, 30000, 32, "f32", True), (256, 512, 9000, 64, "bf16", True),
          (33, 2111, 250007, 4, "f32", True), (256, 3000, 50021, 8, "bf16", True), (512, 3000, 50021, 5, "f32", False)]


@pytest.mark.parametrize("B,N,L,K,storage,tp", SHAPES)
def test_back_to_back(B, N, L, K, storage, tp):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(B)
    dt = torch.bfloat16 if storage == "bf16" else torch.float32
    idx = torch.randint(0, N, (L, K), generator=gen, dtype=torch.int32, device="cuda")
    bias = torch.randn(L, generator=gen, device="cuda")
    row_ptr = torch.arange(B + 1, dtype=torch.int32, device="cuda")
    labels = torch.randint(0, L, (B,), generator=gen, dtype=torch.int32, device="cuda")
    sets = [(torch.randn((N, B) if tp else (B, N), generator=gen, device="cuda").to(dt),
             torch.randn((L, K), generator=gen, device="cuda").to(dt)) for _ in range(3)]
    plan = ops.FFIPlan(idx, N)

    def one(x, W):
        y = (ops.fan_in_sparse_matmul_tp if tp else ops.fan_in_sparse_matmul)(x, idx, W)
        gx, gw, gb = ops._backward(x, idx, W, y, tp, plan=plan, want_bias_grad=True)
        loss, gT = ops.forward_bce(x, idx, W, bias, row_ptr, labels, tp)
        gx2, gw2, gb2 = ops._backward(x, idx, W, gT, tp, plan=plan, want_bias_grad=True, grad_is_transposed=True)
        top, lab = ops.forward_topk(x, idx, W, bias, 3, tp)
        return y, gx, gw, gb, loss, gx2, gw2, gb2, top, lab

    want = []
    for s in sets:
        torch.cuda.synchronize()
        want.append([t.clone() for t in one(*s)])
        torch.cuda.synchronize()
    got = [one(*sets[i % 3]) for i in range(9)]
    for i, outs in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(outs, want[i % 3]))

    x, W = (t.clone() for t in sets[0])
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        one(x, W)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            outs = one(x, W)
        for i in range(6):
            x.copy_(sets[i % 3][0])
            W.copy_(sets[i % 3][1])
            graph.replay()
            assert all(torch.equal(a, b) for a, b in zip(outs, want[i % 3]))
