"""Timed cases of the fixed-fan-in (FFI) sparse layer: what users have it do, over the range they have it done.

Four kinds of call, all through the package's public entry points:

* ``op``    the operator pair (``fan_in_sparse_matmul{,_tp}`` and its ``_grad``) on raw tensors, both layouts, fp32 or
            bf16 storage: how a framework binding calls the library (forward, then both gradients);
* ``layer`` ``FFILayer`` under autograd (fp32, bias), forward and backward of one training step;
* ``step``  the fused training step of an output layer: ``forward_bce`` (loss gradient in the forward's epilogue),
            the backward from the transposed gradient, and optionally ``FusedAdam`` on weights and bias;
* ``topk``  ``forward_topk``: the k best labels per sample, for evaluation (a batch) and for serving (one query).

Sizes are those of the benchmark configurations (L = 670,091 and 501,070 labels, 32,768 / 65,536 / 100,000 hidden
units, fan-in 32 / 64 / 72, batch 32 ... 512) and of the reference's test fixtures (127 x 254 -> 513, fan-in 73).
"""
import math

import torch

import ecml23_sparse_b200 as ffi
from ecml23_sparse_b200 import ops

MAX_WORK = 4.1e9        # B*L*K of the largest listed case
MAX_OUT = 1.28e8        # B*L, likewise


def _case(name, kind, B, N, L, K, dtype="fp32", **more):
    return dict({"name": name, "kind": kind, "B": B, "N": N, "L": L, "K": K, "dtype": dtype}, **more)


def listed():
    return [
        # the reference's ragged test fixture: odd fan-in, odd batch, untransposed op; nothing but latency and launches
        _case("small_odd_op", "op", 127, 254, 513, 73, transposed=False),
        # first layer of the two-layer stack (configuration 1): a small layer inside a large model
        _case("hidden_fp32", "layer", 128, 768, 32768, 32),
        # first layer of the Wikipedia-scale stack (configuration 2), bf16 storage, two batch tiles
        _case("hidden_bf16", "op", 256, 512, 65536, 64, dtype="bf16", transposed=True),
        # serving: one sample's best labels out of 670,091
        _case("query_top5", "topk", 1, 768, 670091, 32, k=5),
        # evaluation: precision at 5 over a test set, a batch at a time
        _case("eval_top5", "topk", 128, 768, 670091, 32, k=5),
        # configuration 0: the output layer alone with the smallest training batch
        _case("layer_batch32", "layer", 32, 768, 670091, 32),
        # the headline: the output layer's forward and backward under autograd
        _case("layer_headline", "layer", 128, 768, 670091, 32),
        # the same layer in a real training loop: fused loss, backward, Adam
        _case("step_headline", "step", 128, 768, 670091, 32, loss="bce", adam=True),
        # the same with bf16 storage of features and weights
        _case("step_headline_bf16", "step", 128, 768, 670091, 32, dtype="bf16", loss="bce", adam=True),
        # output layer of configuration 1: 32,768 hidden activations
        _case("step_wide_fp32", "step", 128, 32768, 670091, 32, loss="bce", adam=False),
        # output layer of configuration 2: 65,536 hidden activations, batch 256, bf16, with Adam
        _case("step_wide_bf16", "step", 256, 65536, 501070, 32, dtype="bf16", loss="bce", adam=True),
        # one rank's label shard of configuration 3 on eight GPUs, with the loss that the task files select
        _case("step_shard_bf16", "step", 512, 100000, 83762, 72, dtype="bf16", loss="squared_hinge", adam=False),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["op", "layer", "step", "step", "topk"])
    dtype = rng.choice(["fp32", "bf16"]) if kind in ("op", "step") else "fp32"
    # batches: round ones and odd ones
    B = _log_int(rng, 1 if kind in ("op", "topk") else 16, 512)
    if B >= 16 and rng.random() < 0.5:
        B = 1 << max(4, min(9, round(math.log2(B))))
    # inputs: embedding widths up to 1024, or the hidden widths of the stacks
    wide = kind in ("op", "step") and rng.random() < 0.3
    N = _log_int(rng, 16384, 100000) if wide else _log_int(rng, 64, 1024)
    if rng.random() < 0.5:
        N = max(64, N // 64 * 64)
    # fan-in: multiples of eight as configured in practice, sometimes any number
    K = _log_int(rng, 8, 80)
    if rng.random() < 0.8:
        K = max(8, K // 8 * 8)
    cap = min(MAX_OUT / B, (MAX_WORK if K % 8 == 0 else MAX_WORK / 4) / (B * K) / (1.5 if N > 1024 else 1.0))
    L = _log_int(rng, 500, max(1000, int(min(700000, cap))))
    case = {"kind": kind, "B": B, "N": N, "L": L, "K": K, "dtype": dtype}
    if kind == "op":
        case["transposed"] = rng.random() < 0.6
    elif kind == "step":
        case["loss"] = rng.choice(["bce", "squared_hinge"])
        case["adam"] = rng.random() < 0.5
    elif kind == "topk":
        case["k"] = rng.choice([1, 3, 5])
    return case


def _table(gen, L, K, N, dev):
    """K distinct inputs per row where that is quick to draw; with replacement (as the layer itself draws its table,
    and practically the same) for wide inputs and for fan-ins near the number of inputs."""
    if N > 1024 or 2 * K > N:
        return torch.randint(0, N, (L, K), generator=gen, dtype=torch.int32, device=dev)
    out = torch.empty((L, K), dtype=torch.int32, device=dev)
    for r0 in range(0, L, 1 << 17):
        keys = torch.rand((min(L, r0 + (1 << 17)) - r0, N), generator=gen, device=dev)
        out[r0:r0 + keys.shape[0]] = torch.topk(keys, K, dim=1, sorted=False).indices.to(torch.int32)
    return out


def _targets(gen, B, L, dev):
    """CSR multi-hot targets: 1 + Poisson(4) draws per sample, Zipf(1.1) over a shuffled label order."""
    counts = 1 + torch.poisson(torch.full((B,), 4.0, device=dev), generator=gen).long().clamp(max=30)
    cdf = torch.cumsum(torch.arange(1, L + 1, dtype=torch.float64, device=dev).pow(-1.1), 0)
    u = torch.rand((B, 31), generator=gen, dtype=torch.float64, device=dev) * cdf[-1]
    labels = torch.randperm(L, generator=gen, device=dev)[torch.searchsorted(cdf, u).clamp(max=L - 1)]
    keep = torch.arange(31, device=dev)[None, :] < counts[:, None]
    flat = torch.unique((labels + L * torch.arange(B, device=dev)[:, None])[keep])
    row_ptr = torch.zeros(B + 1, dtype=torch.int32, device=dev)
    row_ptr[1:] = torch.cumsum(torch.bincount(flat // L, minlength=B), 0).to(torch.int32)
    return row_ptr, (flat % L).to(torch.int32)


def prepare(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    B, N, L, K = case["B"], case["N"], case["L"], case["K"]
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    tp = case.get("transposed", True)

    x = torch.randn((N, B) if tp else (B, N), generator=gen, device=dev)
    if N > 1024:
        x = torch.relu(x)       # hidden activations
    idx = _table(gen, L, K, N, dev)
    W = torch.randn((L, K), generator=gen, device=dev) * (1.0 / K) ** 0.5
    bias = torch.randn(L, generator=gen, device=dev) * 0.1
    x, W = x.to(dtype), W.to(dtype)
    s = {"case": case}
    if case["kind"] == "layer":
        layer = ffi.FFILayer(N, 8, K, seed=0)       # the module, then this case's table, weights and bias
        layer.units, layer.connections = L, L * K
        layer.kernel_indices = idx.view(-1)
        layer.kernel_weights = torch.nn.Parameter(W.view(-1))
        layer.bias = torch.nn.Parameter(bias)
        layer.plan()
        s.update(layer=layer, x=x.t().contiguous().requires_grad_(), g=torch.randn((B, L), generator=gen, device=dev))
    elif case["kind"] == "op":
        ops.get_plan(idx, N)
        s.update(x=x, idx=idx, W=W, g=torch.randn((B, L), generator=gen, device=dev))
    elif case["kind"] == "step":
        row_ptr, labels = _targets(gen, B, L, dev)
        s.update(x=x, idx=idx, W=W, bias=bias, row_ptr=row_ptr, labels=labels, plan=ops.FFIPlan(idx, N),
                 opt=ffi.FusedAdam([W, bias]) if case["adam"] else None)
    else:
        s.update(x=x, idx=idx, W=W, bias=bias)
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "layer":
        layer = s["layer"]
        y = layer(s["x"])
        gx, gw, gb = torch.autograd.grad(y, (s["x"], layer.kernel_weights, layer.bias), s["g"])
        return {"y": y, "grad_x": gx, "grad_w": gw, "grad_bias": gb}
    if case["kind"] == "op":
        if case["transposed"]:
            y = ops.fan_in_sparse_matmul_tp(s["x"], s["idx"], s["W"])
            gx, gw = ops.fan_in_sparse_matmul_grad_tp(s["x"], s["idx"], s["W"], s["g"])
        else:
            y = ops.fan_in_sparse_matmul(s["x"], s["idx"], s["W"])
            gx, gw = ops.fan_in_sparse_matmul_grad(s["x"], s["idx"], s["W"], s["g"])
        return {"y": y, "grad_x": gx, "grad_w": gw}
    if case["kind"] == "step":
        loss, gT = ops.forward_bce(s["x"], s["idx"], s["W"], s["bias"], s["row_ptr"], s["labels"], True,
                                   loss=case["loss"])
        gx, gw, gb = ops._backward(s["x"], s["idx"], s["W"], gT, True, plan=s["plan"], want_bias_grad=True,
                                   grad_is_transposed=True)
        out = {"loss": loss, "grad_x": gx, "grad_w": gw, "grad_bias": gb}
        if s["opt"] is not None:
            s["opt"].step([gw, gb])
            out.update(weights=s["W"], bias=s["bias"], m=s["opt"].m, v=s["opt"].v)
        return out
    val, lab = ops.forward_topk(s["x"], s["idx"], s["W"], s["bias"], case["k"], True)
    return {"values": val, "labels": lab}


def work(case):
    """Each input read once, each output written once; B*L*K multiply-adds per pass of the contraction."""
    B, N, L, K = case["B"], case["N"], case["L"], case["K"]
    e = 2 if case["dtype"] == "bf16" else 4
    nbytes = e * B * N + (e + 4) * L * K            # x, W, idx
    flops = 2 * B * L * K
    if case["kind"] == "topk":
        return {"bytes": nbytes + 4 * L + 8 * B * case["k"], "flops": flops}
    nbytes += 4 * B * N + 4 * L * K                 # grad_x, grad_W
    flops *= 3
    if case["kind"] in ("op", "layer"):
        nbytes += 8 * B * L                         # y, g
    if case["kind"] != "op":
        nbytes += 8 * L                             # bias, grad_bias
    if case.get("adam"):
        nbytes += (16 + e) * L * K + 20 * L         # m, v read and written, W and bias written
        flops += 12 * (L * K + L)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # fp32 accumulation everywhere, also of bf16 products (those are exact in fp32)
    if case["kind"] == "topk":
        return {"rel": 1e-5, "differ": 0.005}       # two labels whose logits round to each other may swap
    if case.get("adam") and case["dtype"] == "bf16":
        return {"rel": 1e-3, "max": 0.01}           # updated bf16 weights: a value may round to its neighbour
    return {"rel": 1e-5}
