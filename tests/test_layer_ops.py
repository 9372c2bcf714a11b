"""Layer operators where the fused kernels do not take a call: values and gradients of the stock operators."""
import pytest
import torch
import torch.nn.functional as F


def _check(dtype, device, N, bias_shape=None, tol=1e-5):
    from oneccl_b200.ops import nn as K

    torch.manual_seed(0)
    x, w = (torch.randn(*s, device=device, dtype=dtype, requires_grad=True) for s in ((5, 16), (N, 16)))
    b = torch.randn(bias_shape or (N,), device=device, dtype=dtype, requires_grad=True)
    dy = torch.randn(5, N, device=device, dtype=dtype)
    y = K.gelu(K.linear(x, w, b, defer_bias=True), b)
    want = F.gelu(F.linear(x, w, b), approximate="tanh")
    torch.testing.assert_close(y, want, rtol=tol, atol=tol)
    for got, ref in zip(torch.autograd.grad(y, [x, w, b], dy), torch.autograd.grad(want, [x, w, b], dy)):
        torch.testing.assert_close(got, ref, rtol=tol, atol=4 * tol)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("N", [8, 13])
def test_deferred_bias_and_gelu_on_cpu(dtype, N):
    """The gradient of a deferred bias arrives once, with every type and width."""
    _check(dtype, "cpu", N)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,N,bias_shape,tol", [
    (torch.float32, 16, None, 1e-5), (torch.float16, 16, None, 4e-3), (torch.bfloat16, 13, None, 3e-2), (torch.bfloat16, 16, (1,), 3e-2),
    (torch.bfloat16, 16, None, 3e-2)])
def test_deferred_bias_and_gelu_on_gpu(dtype, N, bias_shape, tol):
    """Types, widths and bias shapes beside the kernels' own."""
    _check(dtype, "cuda", N, bias_shape, tol)
