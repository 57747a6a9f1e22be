"""Host-side mirror of the reference's Python op binding (sparse/ops/fixed_fan_in_ops.py).

Same function names, argument order and return values as the reference's wrappers
(fixed_fan_in_ops.py:15-28), over torch CUDA tensors instead of TensorFlow tensors:

* ``fan_in_sparse_matmul(features[B,N], lookup[L,K], weights[L,K]) -> [B,L]``
* ``fan_in_sparse_matmul_tp(features[N,B], lookup, weights) -> [B,L]``
* ``fan_in_sparse_matmul_grad(features, lookup, weights, out_grad) -> (feature_grad, weight_grad)``
* ``fan_in_sparse_matmul_grad_tp(...)`` likewise for the transposed layout

and the gradient wiring of fixed_fan_in_ops.py:31-40 (``[feature_grad, None, weight_grad]``)
as an autograd node behind ``ffi_matmul`` / ``ffi_matmul_tp``.
Every call goes through the C ABI of ``libffi_b200.so``; there is no CPU path.  The hot entry points are one native
call each (``csrc/binding.cpp``: checks, output and scratch allocation, launch, autograd node); the rest goes over ctypes.
"""
from __future__ import annotations

import ctypes
import weakref
from typing import Optional

import torch

from . import _lib

_plan_cache: dict = {}
_PLAN_CACHE_MAX = 8


def _stream_ptr(device) -> int:
    return torch.cuda.current_stream(device).cuda_stream


def _native():
    """The native binding; its autograd node asks this module for a table's plan."""
    global _native
    mod = _lib.binding()
    mod.set_get_plan(get_plan)
    _native = lambda: mod  # noqa: E731
    return mod


def _workspace(device, nbytes: int) -> torch.Tensor:
    """Scratch of a call that goes over ctypes, in stream order from torch's allocator (a few kilobytes; the hot entry points
    keep one buffer per stream, csrc/binding.cpp)."""
    return torch.empty(nbytes, dtype=torch.uint8, device=device)


def _check_cuda(name: str, t: torch.Tensor, dtypes) -> torch.Tensor:
    if not isinstance(t, torch.Tensor):
        raise TypeError(f"{name} must be a torch.Tensor")
    if not t.is_cuda:
        raise ValueError(f"{name} must be a CUDA tensor: this library has no CPU path")
    if t.dtype not in dtypes:
        raise TypeError(f"{name} has dtype {t.dtype}, expected one of {dtypes}")
    if t.dim() != 2:
        raise ValueError(f"{name} must have rank 2, got shape {tuple(t.shape)}")
    return t.contiguous()


_INDEX_DTYPES = (torch.int32, torch.uint32) if hasattr(torch, "uint32") else (torch.int32,)


def _as_index(lookup: torch.Tensor) -> torch.Tensor:
    lookup = _check_cuda("lookup", lookup, _INDEX_DTYPES)
    if lookup.dtype != torch.int32:
        lookup = lookup.view(torch.int32)  # values < 2^31 by the reference's contract
    return lookup


class FFIPlan:
    """Transposed (CSR-by-input) index of one lookup table; owns device memory.

    Build one per lookup table and rebuild it whenever the table changes (rewiring).
    """

    def __init__(self, lookup: torch.Tensor, n_in: int):
        lookup = _as_index(lookup)
        self.device = lookup.device
        self.L, self.K = (int(s) for s in lookup.shape)
        self.N = int(n_in)
        handle = ctypes.c_void_p()
        with torch.cuda.device(self.device):
            _lib.check(_lib.load().ffi_plan_create(lookup.data_ptr(), self.L, self.K, self.N,
                                                   _stream_ptr(self.device), ctypes.byref(handle)))
        self._handle = handle
        self.address = handle.value
        self.builds = 1
        self._finalizer = weakref.finalize(self, _lib.load().ffi_plan_destroy, handle)

    def rebuild(self, lookup: torch.Tensor) -> "FFIPlan":
        """Re-derives the plan in place from a table of the same shape whose contents changed (rewiring);
        the index arrays are reused and, from the second rebuild on, nothing is allocated."""
        lookup = _as_index(lookup)
        if tuple(lookup.shape) != (self.L, self.K) or lookup.device != self.device:
            raise ValueError("rebuild needs a table of the plan's shape on the plan's device")
        with torch.cuda.device(self.device):
            _lib.check(_lib.load().ffi_plan_rebuild(self._handle, lookup.data_ptr(), _stream_ptr(self.device)))
        self.builds += 1
        return self

    @property
    def handle(self):
        return self._handle

    def info(self) -> dict:
        vals = [ctypes.c_int64() for _ in range(6)]
        _lib.check(_lib.load().ffi_plan_info(self._handle, *[ctypes.byref(v) for v in vals]))
        names = ("L", "K", "N", "chunk_rows", "n_chunks", "device_bytes")
        return {n: int(v.value) for n, v in zip(names, vals)}

    def export(self, chunked: bool = False):
        """(rowptr[N+1], perm[L*K]) int32 device tensors of the canonical transposed index."""
        rowptr = torch.empty(self.N + 1, dtype=torch.int32, device=self.device)
        perm = torch.empty(self.L * self.K, dtype=torch.int32, device=self.device)
        fn = _lib.load().ffi_plan_export_chunked if chunked else _lib.load().ffi_plan_export
        with torch.cuda.device(self.device):
            _lib.check(fn(self._handle, rowptr.data_ptr(), perm.data_ptr(), _stream_ptr(self.device)))
        return rowptr, perm

    def close(self):
        self._finalizer()


def get_plan(lookup: torch.Tensor, n_in: int) -> FFIPlan:
    """Plan for `lookup`, cached per (storage address, shape, tensor version).

    An in-place update of the table (rewiring) bumps the tensor's version and leads to a
    rebuild of the cached plan in place (`FFIPlan.rebuild`: same object, new contents).  The cache
    keeps a reference to the table so that its address cannot be handed to another tensor while
    the entry lives (at most 8 tables are kept).
    """
    key = (lookup.data_ptr(), lookup.shape, n_in, lookup.get_device())
    hit = _plan_cache.get(key)
    if hit is not None and hit[0] == lookup._version:
        return hit[1]
    if hit is not None:
        plan = hit[1].rebuild(lookup)
        _plan_cache[key] = (lookup._version, plan, lookup)
        return plan
    plan = FFIPlan(lookup, n_in)
    _plan_cache.pop(key, None)
    if len(_plan_cache) >= _PLAN_CACHE_MAX:
        _plan_cache.pop(next(iter(_plan_cache)))
    _plan_cache[key] = (lookup._version, plan, lookup)
    return plan


def clear_caches():
    _plan_cache.clear()
    _native().clear_scratch()


def _forward(features, lookup, weights, bias, transposed: bool) -> torch.Tensor:
    return _native().forward(features, lookup, weights, bias, transposed)


def _backward(features, lookup, weights, out_grad, transposed: bool, plan: Optional[FFIPlan] = None,
              want_feature_grad=True, want_weight_grad=True, want_bias_grad=False, grad_is_transposed=False,
              feature_grad_out: Optional[torch.Tensor] = None):
    """grad_is_transposed: `out_grad` is gT[L][ldg] (from forward_bce / transpose_gradient), not g[B,L].
    feature_grad_out: a contiguous float32 tensor with the number of elements of `features` that
    receives grad_x instead of a fresh allocation (e.g. a slot of a peer-visible buffer)."""
    if want_feature_grad and plan is None:
        plan = get_plan(lookup.contiguous(), features.shape[0 if transposed else 1])
    return _native().backward(features, lookup, weights, out_grad, transposed, plan.address if plan is not None else 0,
                              want_feature_grad, want_weight_grad, want_bias_grad, grad_is_transposed, feature_grad_out)


_LOSS_KINDS = {"bce": _lib.FFI_LOSS_BCE, "squared_hinge": _lib.FFI_LOSS_SQUARED_HINGE, "hinge": _lib.FFI_LOSS_HINGE}


def forward_bce(features, lookup, weights, bias, row_ptr, labels, transposed: bool, total_labels=None,
                label_offset: int = 0, loss: str = "bce", loss_out=None):
    """Forward with the loss gradient fused into its epilogue: returns (loss scalar tensor, gT[L][ldg]).
    `loss` is "bce" (SparseBinaryCrossEntropyLoss), "squared_hinge" (SparseSquaredHingeLoss, the
    one the reference's task files select) or "hinge" (SparseHingeLoss); sparse/metrics.py:132-173.

    The logits are never materialised.  `loss_out` (optional, one fp32 element on the device) receives the
    loss scalar in place, e.g. a slot of the buffer a label-sharded step exchanges."""
    return _native().forward_loss(_LOSS_KINDS[loss], features, lookup, weights, bias, row_ptr, labels, transposed,
                                  total_labels or 0, label_offset, loss_out)


def forward_topk(features, lookup, weights, bias, k: int, transposed: bool, label_offset: int = 0):
    """The k highest logits per sample and their labels, (values[B,k], labels[B,k] int32), in the order
    of tf.nn.top_k, without materialising the logits: what PrecisionAtK (sparse/metrics.py:9-70)
    consumes.  With a sharded label dimension call it per shard (`label_offset` = first label of the
    shard) and merge the candidates with `merge_topk`."""
    return _native().forward_topk(features, lookup, weights, bias, k, transposed, label_offset)


def merge_topk(candidates, k: int):
    """Best k of several shards' (values, labels) candidate lists, again in tf.nn.top_k order."""
    vals = torch.cat([c[0] for c in candidates], dim=1)
    idxs = torch.cat([c[1] for c in candidates], dim=1)
    # value descending, label ascending on ties: sort by label first, then a stable sort by value
    order = torch.argsort(idxs, dim=1, stable=True)
    vals, idxs = torch.gather(vals, 1, order), torch.gather(idxs, 1, order)
    order = torch.argsort(vals, dim=1, descending=True, stable=True)[:, :k]
    return torch.gather(vals, 1, order), torch.gather(idxs, 1, order)


def precision_at_k(top_labels: torch.Tensor, row_ptr: torch.Tensor, labels: torch.Tensor, k: int) -> float:
    """P@k of a batch as PrecisionAtK accumulates it (sparse/metrics.py:58-70): the number of the k
    top-ranked labels that are true labels, summed over the batch, divided by B*k."""
    top = top_labels[:, :k].to(torch.int64).cpu()
    row_ptr, labels = row_ptr.cpu().to(torch.int64), labels.cpu().to(torch.int64)
    correct = 0
    for b in range(top.shape[0]):
        truth = labels[row_ptr[b]:row_ptr[b + 1]]
        correct += int(torch.isin(top[b], truth).sum())
    return correct / (top.shape[0] * k)


def transpose_gradient(out_grad: torch.Tensor, want_bias_grad: bool = False):
    """g[B,L] -> (gT[L][ldg] zero padded in the batch, grad_bias[L] or None): the transposed copy the
    backward kernels read (and the input of the allocation-free grad_x entry point)."""
    out_grad = _check_cuda("out_grad", out_grad, (torch.float32,))
    B, L = out_grad.shape
    lib = _lib.load()
    ldg = int(lib.ffi_transposed_gradient_stride(B))
    gT = torch.empty((L, ldg), dtype=torch.float32, device=out_grad.device)
    gb = torch.empty((L,), dtype=torch.float32, device=out_grad.device) if want_bias_grad else None
    with torch.cuda.device(out_grad.device):
        _lib.check(lib.ffi_transpose_gradient(out_grad.data_ptr(), gT.data_ptr(), gb.data_ptr() if gb is not None else None,
                                              B, L, _stream_ptr(out_grad.device)))
    return gT, gb


# ---- the reference's four wrappers (sparse/ops/fixed_fan_in_ops.py:15-28) -------------

def fan_in_sparse_matmul(features, lookup, weights):
    return _forward(features, lookup, weights, None, False)


def fan_in_sparse_matmul_tp(features, lookup, weights):
    return _forward(features, lookup, weights, None, True)


def fan_in_sparse_matmul_grad(features, lookup, weights, out_grad):
    gx, gw, _ = _backward(features, lookup, weights, out_grad, False)
    return gx, gw


def fan_in_sparse_matmul_grad_tp(features, lookup, weights, out_grad):
    gx, gw, _ = _backward(features, lookup, weights, out_grad, True)
    return gx, gw


# ---- gradient registration (sparse/ops/fixed_fan_in_ops.py:31-40) ---------------------

def ffi_matmul(features, lookup, weights, bias=None):
    """Differentiable FanInSparseMatmul (+ optional fused bias)."""
    return _native().matmul(features, lookup, weights, bias, False)


def ffi_matmul_tp(features, lookup, weights, bias=None):
    """Differentiable FanInSparseMatmulTp (features given as [N,B]) (+ optional fused bias)."""
    return _native().matmul(features, lookup, weights, bias, True)
