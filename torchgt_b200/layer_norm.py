"""``LayerNorm``: ``torch.nn.LayerNorm`` with the same parameters and ``state_dict`` keys whose CUDA fp32
path runs the short-row kernels of ``csrc/layer_norm.cu`` through the node in ``csrc/binding_dense.cpp``
(models/graphormer_dist_node_level.py:301,306,395 are ``nn.LayerNorm(64)`` over 64,000 to 870,000 rows).  Anything
else — CPU tensors, other dtypes, a hidden size the kernels do not cover, no affine parameters, tracing, autocast,
``torch.func`` — is ``torch.nn.LayerNorm`` itself."""
from __future__ import annotations

import ctypes

import torch
from torch.nn.modules import module as _module
from torch.overrides import has_torch_function_variadic

from . import _cabi


def _stream(t: torch.Tensor) -> int:
    return torch.cuda.current_stream(t.device).cuda_stream


_scratch_bytes: dict = {}


def _bwd_scratch(rows: int, hidden: int, device) -> torch.Tensor:
    key = (rows, hidden)
    if key not in _scratch_bytes:
        nb = ctypes.c_size_t()
        _cabi.check(_cabi.load().tgt_layer_norm_bwd_scratch_bytes(rows, hidden, ctypes.byref(nb)))
        _scratch_bytes[key] = nb.value
    return torch.empty(max(_scratch_bytes[key], 16), dtype=torch.uint8, device=device)


def forward_with_stats(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor, eps: float):
    """y and the [rows, 2] (mean, 1/sqrt(var+eps)) the backward needs; x contiguous fp32 on a GPU."""
    hidden = x.shape[-1]
    rows = x.numel() // hidden
    y = torch.empty_like(x)
    stats = torch.empty((rows, 2), dtype=torch.float32, device=x.device)
    with torch.cuda.device(x.device):
        _cabi.check(_cabi.load().tgt_layer_norm_fwd(x.data_ptr(), weight.data_ptr(), bias.data_ptr(), float(eps), rows,
                                                    hidden, y.data_ptr(), stats.data_ptr(), _stream(x)))
    return y, stats


def backward(dy: torch.Tensor, x: torch.Tensor, weight: torch.Tensor, stats: torch.Tensor):
    """dx, dgamma, dbeta from the upstream gradient, the saved input and the forward's statistics."""
    hidden = x.shape[-1]
    rows = x.numel() // hidden
    dx = torch.empty_like(x)
    dgamma = torch.empty(hidden, dtype=torch.float32, device=x.device)
    dbeta = torch.empty(hidden, dtype=torch.float32, device=x.device)
    scratch = _bwd_scratch(rows, hidden, x.device)
    with torch.cuda.device(x.device):
        _cabi.check(_cabi.load().tgt_layer_norm_bwd(dy.data_ptr(), x.data_ptr(), weight.data_ptr(), stats.data_ptr(),
                                                    rows, hidden, dx.data_ptr(), dgamma.data_ptr(), dbeta.data_ptr(),
                                                    scratch.data_ptr(), scratch.numel(), _stream(x)))
    return dx, dgamma, dbeta


def _plain_call(*tensors) -> bool:
    """No tracer, compiler, autocast or tensor subclass wants to see ``F.layer_norm`` itself."""
    return not (torch.compiler.is_compiling() or torch.jit.is_tracing() or torch.is_autocast_enabled("cuda") or
                has_torch_function_variadic(*tensors))


def layer_norm(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor, eps: float = 1e-5) -> torch.Tensor:
    """``F.layer_norm(x, (hidden,), weight, bias, eps)`` over the last dimension."""
    if x.is_cuda and weight is not None and bias is not None and _plain_call(x, weight, bias):
        return _cabi.native().layer_norm(x, weight, bias, eps)
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), weight, bias, eps)


class LayerNorm(torch.nn.LayerNorm):
    """Drop-in for ``nn.LayerNorm(hidden)``: same constructor, parameters and ``state_dict``."""

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        if len(self.normalized_shape) == 1 and self.elementwise_affine and self.bias is not None:
            return layer_norm(x, self.weight, self.bias, self.eps)
        return super().forward(x)


def _bypassable(norm: torch.nn.Module) -> bool:
    """``norm`` is a plain :class:`LayerNorm` whose call nobody observes through module hooks."""
    if type(norm) is not LayerNorm or "forward" in norm.__dict__:
        return False
    hooks = (norm._forward_hooks, norm._forward_pre_hooks, norm._backward_hooks, norm._backward_pre_hooks,
             _module._global_forward_hooks, _module._global_forward_pre_hooks, _module._global_backward_hooks,
             _module._global_backward_pre_hooks)
    return not any(hooks) and len(norm.normalized_shape) == 1 and norm.elementwise_affine and norm.bias is not None


def add_layer_norm(x: torch.Tensor, residual: torch.Tensor, norm: torch.nn.Module, want_sum: bool = True):
    """``(norm(x + residual), x + residual)`` in one kernel each way where ``norm`` allows it.  The second is None
    when ``want_sum`` is false and nothing else needs it."""
    if (x.is_cuda and x.dtype == residual.dtype and x.shape == residual.shape and _bypassable(norm) and
            _plain_call(x, residual, norm.weight, norm.bias)):
        return _cabi.native().add_layer_norm(x, residual, norm.weight, norm.bias, norm.eps, want_sum)
    x = x + residual
    return norm(x), x
