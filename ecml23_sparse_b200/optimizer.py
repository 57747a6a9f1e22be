"""Fused Adam on the flat FFI weight vector.

Mirror of ``SparseAdam`` (sparse/optimizer.py:9-23), i.e. ``keras.optimizers.Adam`` with its
defaults as used at run.py:126 (lr 1e-3, beta 0.9/0.999, epsilon 1e-7, no amsgrad): one fused
launch for all parameters instead of Keras' chain of elementwise ops.  ``zero_moments`` is the
moment reset that ``SparseAdam.update_sparse`` performs at rewired positions
(custom_layer.py:20-30).
"""
from __future__ import annotations

import torch

from . import ops


class FusedAdam:
    def __init__(self, params, lr: float = 1e-3, beta_1: float = 0.9, beta_2: float = 0.999, epsilon: float = 1e-7):
        self.params = [p for p in params]
        for p in self.params:
            if not p.is_cuda or p.dtype not in (torch.float32, torch.bfloat16) or not p.is_contiguous():
                raise ValueError("FusedAdam needs contiguous float32/bfloat16 CUDA parameters")
        self.lr, self.beta_1, self.beta_2, self.epsilon = lr, beta_1, beta_2, epsilon
        self.iterations = 0
        self.m = [torch.zeros(p.shape, dtype=torch.float32, device=p.device) for p in self.params]
        self.v = [torch.zeros(p.shape, dtype=torch.float32, device=p.device) for p in self.params]

    def step(self, grads=None):
        """Applies one update; `grads` defaults to each parameter's `.grad`."""
        self.iterations += 1
        todo = []
        for j, p in enumerate(self.params):
            g = grads[j] if grads is not None else p.grad
            if g is not None:
                todo.append((p.data if isinstance(p, torch.nn.Parameter) else p, self.m[j], self.v[j], g))
        if todo:
            ops._native().adam_step(todo, self.lr, self.beta_1, self.beta_2, self.epsilon, self.iterations)

    def zero_moments(self, index: int, locations: torch.Tensor):
        """Zero m and v of parameter `index` at flat positions `locations`."""
        self.m[index].view(-1)[locations] = 0
        self.v[index].view(-1)[locations] = 0
