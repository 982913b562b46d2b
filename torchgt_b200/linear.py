"""``Linear``: ``torch.nn.Linear`` with the same parameters and ``state_dict`` keys for narrow fp32 layers over many
rows (the models' 64 x 64 projections and FFN layers over 4,000 to 870,000 rows), and the blocks the models build of it.  The
nodes are in ``csrc/binding_dense.cpp``: full fp32 products and input gradients run on the tensor cores from three bf16 pieces
per value (``csrc/linear_mma.cu``; few rows: ``csrc/linear_rows.cu``), or as the library's GEMM, by rules on rows, widths and
whether the caller allows TF32 (there, with the times of both sides; with TF32 allowed single layers are the library's, and blocks
but the narrow ones); weight and bias gradients run ``csrc/linear_wgrad.cu``.  CPU tensors, other dtypes, inputs that are
not a multiple of 64 wide and outputs that are not a multiple of 4 wide are ``torch.nn.functional.linear``, and so is whatever
is traced, compiled, autocast or transformed by ``torch.func``."""
from __future__ import annotations

import ctypes

import torch
from torch.nn import functional as F
from torch.nn.modules import module as _module
from torch.overrides import has_torch_function_variadic

from . import _cabi

_scratch_bytes: dict = {}


def _aligned(t: torch.Tensor) -> torch.Tensor:
    """``t`` itself, or a copy when it is a view that starts off a 16-byte boundary (the kernels load 16 bytes
    at a time)."""
    return t if t.data_ptr() % 16 == 0 else t.clone()


def wgrad(dy: torch.Tensor, x: torch.Tensor, with_bias: bool = True):
    """``dy.t() @ x`` and ``dy.sum(0)`` for contiguous fp32 ``dy`` [rows, out] and ``x`` [rows, in] on a GPU."""
    dy, x = _aligned(dy), _aligned(x)
    rows, out_features = dy.shape
    in_features = x.shape[1]
    key = (rows, in_features, out_features)
    if key not in _scratch_bytes:
        nb = ctypes.c_size_t()
        _cabi.check(_cabi.load().tgt_linear_wgrad_scratch_bytes(rows, in_features, out_features, ctypes.byref(nb)))
        _scratch_bytes[key] = nb.value
    scratch = torch.empty(max(_scratch_bytes[key], 16), dtype=torch.uint8, device=dy.device)
    dw = torch.empty((out_features, in_features), dtype=torch.float32, device=dy.device)
    db = torch.empty(out_features, dtype=torch.float32, device=dy.device) if with_bias else None
    with torch.cuda.device(dy.device):
        _cabi.check(_cabi.load().tgt_linear_wgrad(dy.data_ptr(), x.data_ptr(), rows, in_features, out_features,
                                                  dw.data_ptr(), db.data_ptr() if with_bias else None,
                                                  scratch.data_ptr(), scratch.numel(),
                                                  torch.cuda.current_stream(dy.device).cuda_stream))
    return dw, db


def plain_call(*tensors) -> bool:
    """No tracer, compiler, autocast or tensor subclass wants to see PyTorch's own operation."""
    return not (torch.compiler.is_compiling() or torch.jit.is_tracing() or torch.is_autocast_enabled("cuda") or
                has_torch_function_variadic(*tensors))


def linear(x: torch.Tensor, weight: torch.Tensor, bias) -> torch.Tensor:
    """``F.linear(x, weight, bias)``."""
    if x.is_cuda and plain_call(x, weight, bias):
        return _cabi.native().linear(x, weight, bias)
    return F.linear(x, weight, bias)


class Linear(torch.nn.Linear):
    """Drop-in for ``nn.Linear``: same constructor, parameters and ``state_dict``."""

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        return linear(x, self.weight, self.bias)


def unobserved(module: torch.nn.Module, kind: type) -> bool:
    """``module`` is a plain ``kind`` whose call nobody observes through module hooks."""
    if type(module) is not kind or "forward" in module.__dict__:
        return False
    return not any((module._forward_hooks, module._forward_pre_hooks, module._backward_hooks, module._backward_pre_hooks,
                    _module._global_forward_hooks, _module._global_forward_pre_hooks, _module._global_backward_hooks,
                    _module._global_backward_pre_hooks))


def plain_modules(*pairs) -> bool:
    """Every (module, kind) is :func:`unobserved`."""
    if any((_module._global_forward_hooks, _module._global_forward_pre_hooks, _module._global_backward_hooks,
            _module._global_backward_pre_hooks)):
        return False
    for module, kind in pairs:
        own = module.__dict__
        if type(module) is not kind or "forward" in own or own["_forward_hooks"] or own["_forward_pre_hooks"] or \
                own["_backward_hooks"] or own["_backward_pre_hooks"]:
            return False
    return True


def linear3(x: torch.Tensor, a: torch.nn.Module, b: torch.nn.Module, c: torch.nn.Module):
    """``a(x), b(x), c(x)``: one node that reads ``x`` once each way where the three are plain layers of equal shape."""
    layers = (a, b, c)
    if x.is_cuda and all(unobserved(m, Linear) and plain_call(x, m.weight, m.bias) for m in layers):
        return _cabi.native().linear3(x, [m.weight for m in layers], [m.bias for m in layers])
    return a(x), b(x), c(x)


def feed_forward(x: torch.Tensor, first: torch.nn.Module, second: torch.nn.Module, activation: str, residual=None):
    """``(residual +) second(act(first(x)))`` with ``activation`` "relu" or "gelu" (exact), one node whose activation is
    part of the products' kernels, or None where the caller has to go through the modules."""
    if not (x.is_cuda and unobserved(first, Linear) and unobserved(second, Linear) and first.bias is not None and
            second.bias is not None and plain_call(x, first.weight, first.bias) and
            not has_torch_function_variadic(second.weight, second.bias, residual)):
        return None
    return _cabi.native().feed_forward(x, first.weight, first.bias, second.weight, second.bias, activation, residual)


def passes_through(dropout: torch.nn.Module) -> bool:
    """``dropout`` returns its input as it is, and nobody observes the call."""
    return unobserved(dropout, torch.nn.Dropout) and (not dropout.training or dropout.p == 0.0)


def embedding_sum(embedding: torch.nn.Module, ids: torch.Tensor) -> torch.Tensor:
    """``embedding(ids).sum(dim=-2)``; the gathered vectors are never stored (csrc/embedding_sum.cu)."""
    if (ids.is_cuda and unobserved(embedding, torch.nn.Embedding) and embedding.max_norm is None and not embedding.sparse and
            not embedding.scale_grad_by_freq and plain_call(ids, embedding.weight, None)):
        padding = -1 if embedding.padding_idx is None else embedding.padding_idx
        return _cabi.native().embedding_sum(embedding.weight, ids, padding)
    return embedding(ids).sum(dim=-2)
