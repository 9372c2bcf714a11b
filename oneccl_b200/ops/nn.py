"""Fused layer pieces for the training path (bf16 activations, fp32 math); kernels in ``csrc/gpu/nn_kernels.cu`` and
``embedding_kernels.cu``, autograd functions in ``oneccl_b200/torch_ops/nn_ops.cpp``:

* ``layer_norm`` / ``add_layer_norm``: LayerNorm whose backward produces the input gradient and the
  weight / bias gradients from one read of the activations; the ``add_`` form also performs the residual
  addition in front of it (and adds the residual branch's gradient inside the backward kernel);
* ``linear``: cuBLAS matmuls, with the bias gradient by a column sum or left to the next operator;
* ``split_qkv``: views of a packed QKV projection for the attention call, whose backward assembles the
  packed gradient and sums it over the rows in one pass;
* ``gelu``: tanh-form GELU; ``mlp``: two linear layers with a GELU between them, which runs inside the products
  (``csrc/gpu/gemm_mlp.cu``); ``embed``: token plus position embedding.

The kernel that produces the gradient of a linear layer's output can sum the bias gradient on the way.  ``linear(...,
defer_bias=True)`` leaves it to the operator that consumes the output and is given the bias: ``add_layer_norm(...,
res_bias=b)``, ``split_qkv(..., bias=b)``, ``gelu(u, b)``.

A parameter may carry a gradient sink (``oneccl_b200.torch_ops.GradSink``, set by ``DataParallel``): its gradient is then
written into the flat gradient buffer by the operator itself and autograd gets none to accumulate.

Shapes the kernels do not cover (LayerNorm width not a multiple of 8, below 256 or above 2048, non-bf16, CPU)
fall back to the equivalent PyTorch ops."""
from __future__ import annotations

import torch
import torch.nn.functional as F

from ..torch_ops import native


def layer_norm(x, weight, bias, eps: float = 1e-5):
    y = native().add_layer_norm(x, None, weight, bias, eps)
    return F.layer_norm(x, (x.shape[-1],), weight, bias, eps) if y is None else y


def add_layer_norm(x, res, weight, bias, eps: float = 1e-5, res_bias=None):
    """Returns (LayerNorm(x + res), x + res).  ``res_bias``: the bias of the linear layer that produced ``res`` with
    ``defer_bias``; only where ``fused_width(x)`` holds."""
    if res is None:
        return layer_norm(x, weight, bias, eps), x
    out = native().add_layer_norm(x, res, weight, bias, eps, res_bias)
    if out is None:
        assert res_bias is None, "a deferred bias gradient needs the fused LayerNorm"
        s = x + res
        return F.layer_norm(s, (s.shape[-1],), weight, bias, eps), s
    return out


def fused_width(x, ln) -> bool:
    """Whether ``add_layer_norm`` of ``x`` with the parameters of ``ln`` runs on the fused kernels (and may so take over
    bias gradients)."""
    return native().layer_norm_ok(x, None, ln.weight, ln.bias)


def colsum(dy2: torch.Tensor) -> torch.Tensor:
    """Sum over the rows of a contiguous [rows, N] bf16 matrix (fp32 accumulation, fixed order)."""
    return native().colsum(dy2)


def linear(x, weight, bias, defer_bias: bool = False, last_use: bool = True):
    """``last_use=False``: the weight is used again closer to the model's input (a tied embedding), which then
    contributes the last part of its gradient."""
    if bias is None and getattr(weight, "_grad_sink", None) is None:
        return F.linear(x, weight)
    y = native().linear(x, weight, bias, not defer_bias, last_use)
    if y is None:  # the operator that consumes the output returns a deferred bias gradient in any case
        return F.linear(x, weight, bias.detach() if defer_bias and bias is not None else bias)
    return y


def gelu(u, bias):
    """tanh-form GELU of ``u``, the output of a ``linear(..., bias, defer_bias=True)``."""
    y = native().bias_gelu(u, bias)
    if y is None:  # adds nothing, but hands the bias its gradient
        return F.gelu(u + (bias - bias.detach()).to(u.dtype), approximate="tanh")
    return y


def mlp(x, w1, b1, w2, b2):
    """``gelu(x @ w1.T + b1) @ w2.T + b2`` with the tanh-form GELU and its gradient inside the products where that is expected to
    be faster, else as ``linear``, ``gelu``, ``linear``.  ``b2``'s gradient is left to the operator that consumes the output."""
    y = native().mlp(x, w1, b1, w2, b2, True)
    if y is None:
        return linear(gelu(linear(x, w1, b1, defer_bias=True), b1), w2, b2, defer_bias=True)
    return y


def split_qkv(qkv: torch.Tensor, n_head: int, bias=None):
    """[B, S, 3 * D] -> q, k, v as [B, H, S, D / H] views."""
    out = native().split_qkv(qkv, n_head, bias)
    if out is None:
        assert bias is None, "a deferred bias gradient needs the fused split"
        B, S, D3 = qkv.shape
        q, k, v = qkv.view(B, S, 3, n_head, D3 // 3 // n_head).permute(2, 0, 3, 1, 4)
        return q, k, v
    return out


def embed(idx, tokens, positions):
    """tokens[idx] + positions[: S] for ids [B, S].  An id outside the table makes its row NaN; as the GPU finds out, a later
    ``embed``, its backward or ``GraphedTrainStep`` call raises the IndexError."""
    if idx.dim() == 2 and idx.shape[1] > positions.shape[0]:
        raise IndexError(f"{idx.shape[1]} positions, but a table of {positions.shape[0]}")
    x = native().embed(idx, tokens, positions)
    if x is None:
        return F.embedding(idx, tokens) + positions[: idx.shape[1]]
    return x
