"""Training-step kernels next to the gradient collective: fused softmax
cross-entropy (logits become their own gradient in place), squared gradient
norm and flat fused AdamW with fp32 master weights.  All three are native
kernels from ``csrc/gpu/train_kernels.cu``; ``launch_count`` (kernels launched by this
package's training and layer operators so far) lets callers report how many of them ran."""
from __future__ import annotations

import torch

from .. import _lib
from ..dtypes import torch_to_ccl
from ..torch_ops import native
from .device_group import _stream_ptr

# the stored logit gradient assumes d(loss) = 1; True multiplies it by the upstream gradient
scale_by_upstream = False

_py_launches = 0


def _bump(n=1):
    global _py_launches
    _py_launches += n


def __getattr__(name):
    if name == "launch_count":
        return _py_launches + native().launch_count()
    raise AttributeError(name)


def softmax_cross_entropy(logits: torch.Tensor, targets: torch.Tensor, vocab: int | None = None) -> torch.Tensor:
    """Mean cross-entropy over the rows of ``logits`` ([rows, cols] bf16; only the
    first ``vocab`` columns are classes, the rest is alignment padding).  ``logits``
    is consumed: it holds the gradient afterwards.  ``targets`` int64."""
    assert logits.dtype == torch.bfloat16 and logits.dim() == 2 and logits.stride(1) == 1
    return native().softmax_xent(logits, targets, logits.shape[1] if vocab is None else vocab, scale_by_upstream)


_partials = {}


def sq_norm(flat_grad: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
    """out[0] += sum(flat_grad**2) (out: 1-element fp32 device tensor).  Two deterministic
    stages (fixed summation order), so every data-parallel rank computes the same bits."""
    lib = _lib.load()
    key = flat_grad.device
    if key not in _partials:
        _partials[key] = torch.empty(1024, dtype=torch.float32, device=flat_grad.device)
    _lib.check(lib.cclx_sq_norm(flat_grad.data_ptr(), flat_grad.numel(), torch_to_ccl(flat_grad.dtype),
                                out.data_ptr(), _partials[key].data_ptr(), _stream_ptr()))
    _bump(2)
    return out


class FlatAdamW:
    """AdamW over one flat parameter buffer.

    ``model_flat`` (bf16) is what the model's parameters are views of; the
    optimizer keeps fp32 master / m / v copies and rewrites ``model_flat`` in
    the same kernel.  Elements ``[0, n_decay)`` receive weight decay.  The
    gradient is read in its own dtype (bf16 buckets are never widened in
    memory).  ``max_norm`` > 0 enables clipping by the global norm, which is
    computed on the device and consumed on the device (no host sync).
    ``device_step=True`` keeps the step number (bias corrections) in a device word that the
    kernel sequence increments itself, which is what a step replayed from a CUDA graph needs.
    """

    def __init__(self, model_flat: torch.Tensor, n_decay: int, lr=3e-4, betas=(0.9, 0.95), eps=1e-8,
                 weight_decay=0.1, max_norm: float = 1.0, device_step: bool = False):
        self.model_flat = model_flat if model_flat.dtype == torch.bfloat16 else None
        self.master = model_flat.detach().to(torch.float32).clone()
        self._fp32_model = model_flat if model_flat.dtype == torch.float32 else None
        self.m = torch.zeros_like(self.master)
        self.v = torch.zeros_like(self.master)
        self.n_decay = int(n_decay)
        self.lr, self.betas, self.eps, self.weight_decay, self.max_norm = lr, betas, eps, weight_decay, max_norm
        self.step_count = 0
        self._norm = torch.zeros(1, dtype=torch.float32, device=model_flat.device)
        self._counter = torch.zeros(1, dtype=torch.int32, device=model_flat.device)  # arrivals of the norm's blocks
        self._step_dev = torch.zeros(1, dtype=torch.int32, device=model_flat.device) if device_step else None

    def step(self, flat_grad: torch.Tensor, grad_scale: float = 1.0):
        self.step_count += 1
        native().adamw_step(self.master, flat_grad, self.m, self.v, self.model_flat, self.n_decay, self.lr, *self.betas, self.eps,
                            self.weight_decay, self.step_count, grad_scale, self.max_norm, self._norm, self._counter, self._step_dev)
        if self._fp32_model is not None:
            self._fp32_model.copy_(self.master)

    def grad_norm(self) -> torch.Tensor:
        return self._norm.sqrt()
