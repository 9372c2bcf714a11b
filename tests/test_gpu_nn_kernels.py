"""Fused LayerNorm (+ residual), bias-gradient column sums and the packed QKV gradient against PyTorch fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [256, 768, 1024])
@pytest.mark.parametrize("rows", [1, 37, 4100])
@pytest.mark.parametrize("residual", [False, True])
def test_layer_norm_forward_backward(D, rows, residual):
    from oneccl_b200.ops.nn import add_layer_norm, layer_norm

    g = torch.Generator(device="cuda").manual_seed(D + rows)
    x = torch.randn(rows, D, generator=g, device="cuda").to(torch.bfloat16)
    r = torch.randn(rows, D, generator=g, device="cuda").to(torch.bfloat16)
    w = (1 + 0.1 * torch.randn(D, generator=g, device="cuda")).to(torch.bfloat16)
    b = (0.1 * torch.randn(D, generator=g, device="cuda")).to(torch.bfloat16)
    dy = torch.randn(rows, D, generator=g, device="cuda").to(torch.bfloat16)
    dsum = torch.randn(rows, D, generator=g, device="cuda").to(torch.bfloat16)

    xs = [t.clone().requires_grad_(True) for t in (x, r, w, b)]
    if residual:
        y, s = add_layer_norm(xs[0], xs[1], xs[2], xs[3])
        torch.autograd.backward([y, s], [dy, dsum])
    else:
        y = layer_norm(xs[0], xs[2], xs[3])
        y.backward(dy)
    # fp32 reference on the same bf16 inputs (the residual sum is rounded to bf16, as the kernel keeps it)
    ref = [t.float().clone().requires_grad_(True) for t in (x, r, w, b)]
    tot = (ref[0] + ref[1]).to(torch.bfloat16).float() if residual else ref[0]
    if residual:
        tot = ref[0] + ref[1] + ((ref[0] + ref[1]).to(torch.bfloat16).float() - (ref[0] + ref[1])).detach()
    yr = torch.nn.functional.layer_norm(tot, (D,), ref[2], ref[3])
    if residual:
        torch.autograd.backward([yr, tot], [dy.float(), dsum.float()])
    else:
        yr.backward(dy.float())
    torch.cuda.synchronize()
    torch.testing.assert_close(y.float(), yr, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(xs[0].grad.float(), ref[0].grad, rtol=2e-2, atol=3e-2)
    if residual:
        assert torch.equal(xs[0].grad, xs[1].grad)
        torch.testing.assert_close(s.float(), tot, rtol=0, atol=0)
    scale = max(1.0, rows ** 0.5)
    torch.testing.assert_close(xs[2].grad.float(), ref[2].grad, rtol=2e-2, atol=2e-2 * scale)
    torch.testing.assert_close(xs[3].grad.float(), ref[3].grad, rtol=2e-2, atol=2e-2 * scale)


def test_layer_norm_falls_back_for_other_widths():
    from oneccl_b200.ops.nn import layer_norm

    x = torch.randn(5, 128, device="cuda").to(torch.bfloat16)
    w = torch.ones(128, device="cuda", dtype=torch.bfloat16)
    b = torch.zeros(128, device="cuda", dtype=torch.bfloat16)
    torch.testing.assert_close(layer_norm(x, w, b), torch.nn.functional.layer_norm(x, (128,), w, b))


@pytest.mark.parametrize("rows,N", [(1, 8), (33, 264), (8192, 3072)])
def test_linear_bias_gradient(rows, N):
    from oneccl_b200.ops.nn import linear

    g = torch.Generator(device="cuda").manual_seed(rows)
    K = 64
    x = torch.randn(rows, K, generator=g, device="cuda").to(torch.bfloat16).requires_grad_(True)
    w = (0.1 * torch.randn(N, K, generator=g, device="cuda")).to(torch.bfloat16).requires_grad_(True)
    b = torch.zeros(N, device="cuda", dtype=torch.bfloat16).requires_grad_(True)
    dy = torch.randn(rows, N, generator=g, device="cuda").to(torch.bfloat16)
    linear(x, w, b).backward(dy)
    xr, wr, br = (t.detach().clone().requires_grad_(True) for t in (x, w, b))
    torch.nn.functional.linear(xr, wr, br).backward(dy)
    torch.cuda.synchronize()
    torch.testing.assert_close(b.grad.float(), dy.float().sum(0), rtol=1e-2, atol=1e-2 * max(1.0, rows ** 0.5))
    torch.testing.assert_close(x.grad, xr.grad)
    torch.testing.assert_close(w.grad, wr.grad)


def test_split_qkv_gradient_matches_unbind():
    from oneccl_b200.ops.nn import split_qkv

    B, S, H, dh = 2, 128, 4, 64
    g = torch.Generator(device="cuda").manual_seed(0)
    qkv = torch.randn(B, S, 3 * H * dh, generator=g, device="cuda").to(torch.bfloat16)
    outs = []
    for fused in (True, False):
        t = qkv.clone().requires_grad_(True)
        if fused:
            q, k, v = split_qkv(t, H)
        else:
            q, k, v = t.view(B, S, 3, H, dh).permute(2, 0, 3, 1, 4)
        a = torch.nn.functional.scaled_dot_product_attention(q, k, v, is_causal=True)
        a.sum().backward()
        outs.append((a.detach(), t.grad))
    torch.cuda.synchronize()
    assert torch.equal(outs[0][0], outs[1][0])
    torch.testing.assert_close(outs[0][1], outs[1][1], rtol=0, atol=0)


def test_gpt2_fused_ops_match_stock_modules():
    from oneccl_b200.models.gpt2 import GPT2, GPT2Config

    cfg = GPT2Config(2, 4, 256, 64, 1000)
    torch.manual_seed(0)
    m = GPT2(cfg, fused_ops=True).cuda().to(torch.bfloat16)
    idx = torch.randint(0, cfg.vocab, (4, 64), device="cuda")
    tgt = torch.randint(0, cfg.vocab, (4, 64), device="cuda")
    grads = []
    losses = []
    for fused in (True, False):
        m.fused_ops = fused
        m.zero_grad(set_to_none=True)
        loss = m(idx, tgt)
        loss.backward()
        losses.append(float(loss.detach()))
        grads.append(torch.cat([p.grad.float().flatten() for p in m.parameters()]))
    assert abs(losses[0] - losses[1]) < 2e-2
    cos = torch.nn.functional.cosine_similarity(grads[0], grads[1], dim=0).item()
    assert cos > 0.99, cos


def test_data_parallel_gradient_sinks_match_autograd():
    """Linear layers accumulate their weight gradients straight into DataParallel's flat buffer (GEMM with
    beta = 1, no autograd accumulation): same gradients as the plain module, every bucket still fires."""
    from oneccl_b200.models.gpt2 import GPT2, GPT2Config
    from oneccl_b200.ops.device_group import DeviceGroup
    from oneccl_b200.parallel.ddp import DataParallel

    cfg = GPT2Config(2, 4, 256, 64, 1000)
    torch.manual_seed(0)
    plain = GPT2(cfg, fused_ops=True).cuda().to(torch.bfloat16)
    torch.manual_seed(0)
    wrapped = GPT2(cfg, fused_ops=True).cuda().to(torch.bfloat16)
    group = DeviceGroup.emulated(1, heap_bytes=64 << 20, staging_bytes=1 << 20)
    ddp = DataParallel(wrapped, group, bucket_mb=0.5)
    idx = torch.randint(0, cfg.vocab, (4, 64), device="cuda")
    tgt = torch.randint(0, cfg.vocab, (4, 64), device="cuda")
    for _ in range(2):  # the second pass checks that zero_grad re-arms everything
        plain.zero_grad(set_to_none=True)
        plain(idx, tgt).backward()
        ddp.zero_grad()
        ddp(idx, tgt).backward()
        ddp.finish()
        torch.cuda.synchronize()
        assert all(b.pending == 0 for b in ddp.buckets)
        for (n, a), (_, b) in zip(plain.named_parameters(), wrapped.named_parameters()):
            torch.testing.assert_close(b.grad.float(), a.grad.float(), rtol=2e-2, atol=2e-3, msg=n)
    group.close()


def test_data_parallel_with_the_gelu_inside_the_products():
    """Batches large enough for the MLP's own kernels: weight gradients beside backward, deferred bias sums, accumulation over two
    passes, a graphed step; against the plain module's autograd."""
    from oneccl_b200.models.gpt2 import GPT2, GPT2Config
    from oneccl_b200.ops.device_group import DeviceGroup
    from oneccl_b200.parallel.ddp import DataParallel, GraphedTrainStep
    from oneccl_b200.torch_ops import native

    cfg = GPT2Config(2, 4, 256, 512, 1000)
    models = []
    for _ in range(2):
        torch.manual_seed(0)
        models.append(GPT2(cfg, fused_ops=True).cuda().to(torch.bfloat16))
    plain, wrapped = models
    block, x = plain.blocks[0], torch.zeros(4096, 256, dtype=torch.bfloat16, device="cuda")
    assert native().mlp(x, block.fc.weight, block.fc.bias, block.fc2.weight, block.fc2.bias) is not None
    idx, tgt = (torch.randint(0, cfg.vocab, (8, 512), device="cuda") for _ in range(2))
    group = DeviceGroup.emulated(1, heap_bytes=64 << 20, staging_bytes=1 << 20)
    ddp = DataParallel(wrapped, group, bucket_mb=0.25)

    def compare(passes):
        plain.zero_grad(set_to_none=True)
        for _ in range(passes):
            plain(idx, tgt).backward()
        torch.cuda.synchronize()
        assert all(b.pending == 0 for b in ddp.buckets)
        for (n, a), (_, b) in zip(plain.named_parameters(), wrapped.named_parameters()):
            # the same kernels: they differ where autograd rounds a second contribution before it adds it
            off = float((b.grad.double() - a.grad.double()).norm() / a.grad.double().norm())
            assert off <= 2.0**-7, (n, off)

    for _ in range(2):
        ddp.begin_step()
        ddp(idx, tgt).backward()
        ddp.finish()
        compare(1)
    ddp.zero_grad()
    for _ in range(2):
        ddp(idx, tgt).backward()
    ddp.finish()
    compare(2)
    step = GraphedTrainStep(ddp, ddp.make_optimizer(device_step=True, lr=0.0, weight_decay=0.0), idx, tgt)
    step(idx, tgt)
    compare(1)
    group.close()


def test_mlp_reports_its_gradients_in_the_order_of_the_operators_of_their_own():
    """Whether a rank's batch is large enough for the products with the GELU inside must not show in the order of its buckets."""
    from oneccl_b200.ops import nn as K
    from oneccl_b200.torch_ops import native

    g = torch.Generator(device="cuda").manual_seed(8)
    rows, D, N = 4608, 64, 1024
    x, dy = (torch.randn(rows, D, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    params = {"w1": (N, D), "b1": (N,), "w2": (D, N), "b2": (D,)}
    params = {k: torch.nn.Parameter((torch.randn(*s, generator=g, device="cuda") * 0.1).to(torch.bfloat16)) for k, s in params.items()}
    seen = []
    for name, p in params.items():
        p._grad_sink = native().GradSink(torch.zeros_like(p), lambda name=name: seen.append(name))
    w1, b1, w2, b2 = params.values()
    orders, grads = [], []
    for y in (native().mlp(x, w1, b1, w2, b2), K.linear(K.gelu(K.linear(x, w1, b1, defer_bias=True), b1), w2, b2, defer_bias=True)):
        seen.clear()
        for p in params.values():
            p._grad_sink.fresh = True
        y.backward(dy)
        orders.append(list(seen))
        grads.append([p._grad_sink.grad.clone() for p in (w1, b1, w2)])
    assert orders[0] == orders[1] and sorted(orders[0]) == ["b1", "w1", "w2"]
    for a, b in zip(*grads):  # each side rounds the sums, the activations and their gradient to bf16 once
        assert float((a.double() - b.double()).norm() / b.double().norm()) <= 2.0**-7


@pytest.mark.parametrize("rows,D,N,inside", [(4096, 256, 1024, True), (2048, 512, 2048, True), (300, 64, 16384, False),
                                             (666, 64, 5120, False), (8192, 64, 3064, False), (2048, 64, 4104, False)])
def test_mlp_keeps_to_the_operators_of_their_own_where_they_are_faster(rows, D, N, inside):
    """Rows of tiles that are mostly padding, and rows of the result that begin between sectors."""
    from oneccl_b200.torch_ops import native

    x, w1, b1, w2, b2 = (torch.zeros(*s, dtype=torch.bfloat16, device="cuda") for s in ((rows, D), (N, D), (N,), (D, N), (D,)))
    assert native().mlp(x, w1, b1, w2, b2) is not None
    assert (native().mlp(x, w1, b1, w2, b2, True) is not None) == inside


def test_mlp_under_autocast_to_another_type():
    """The products with the GELU inside know bf16 alone: under fp16 autocast the operators of their own run, under bf16 both agree."""
    from oneccl_b200.ops import nn as K
    from oneccl_b200.torch_ops import native

    g = torch.Generator(device="cuda").manual_seed(9)
    x, w1, b1, w2, b2 = ((torch.randn(*s, generator=g, device="cuda") * 0.1).to(torch.bfloat16)
                         for s in ((4608, 64), (1024, 64), (1024,), (64, 1024), (64,)))
    with torch.autocast("cuda", torch.float16):
        assert native().mlp(x, w1, b1, w2, b2) is None
        assert K.mlp(x, w1, b1, w2, b2).dtype == torch.float16
    with torch.autocast("cuda", torch.bfloat16):
        inside = native().mlp(x, w1, b1, w2, b2)
    assert torch.equal(inside, native().mlp(x, w1, b1, w2, b2))


@pytest.mark.parametrize("shape", [(4608, 64, 1024, 136), (1999, 1032, 2056, 8), (2305, 768, 3072, 768), (3, 600, 264, 2200, 64)])
def test_mlp(shape):
    """Two linear layers with the GELU inside the products against the same chain of operators of their own, and both against
    64 bits: partial tiles in every dimension, K of one step, several leading dimensions."""
    from oneccl_b200.ops import nn as K
    from oneccl_b200.torch_ops import native

    lead, (D, N, O) = (shape[:-3], shape[-3:])
    g = torch.Generator(device="cuda").manual_seed(3)

    def make(*s, scale=1.0):
        return (torch.randn(*s, generator=g, device="cuda") * scale).to(torch.bfloat16)

    x, w1, b1, w2, b2 = make(*lead, D), make(N, D, scale=D**-0.5), make(N), make(O, N, scale=N**-0.5), make(O)
    dy = make(*lead, O)
    ins = [t.requires_grad_(True) for t in (x, w1, b1, w2)]

    def chain():
        return K.linear(K.gelu(K.linear(x, w1, b1, defer_bias=True), b1), w2, b2, defer_bias=True)

    fused = native().mlp(x, w1, b1, w2, b2)
    assert fused is not None
    outs = []
    for y in (fused, chain()):
        outs.append((y.detach(), *torch.autograd.grad(y, ins, dy)))
    xd, w1d, b1d, w2d = (t.detach().double().requires_grad_(True) for t in ins)
    yd = torch.nn.functional.gelu(xd @ w1d.t() + b1d, approximate="tanh") @ w2d.t() + b2.double()
    exact = (yd.detach(), *torch.autograd.grad(yd, (xd, w1d, b1d, w2d), dy.double()))
    for a, b, e in zip(*outs, exact):
        assert a.shape == b.shape == e.shape and a.dtype == b.dtype
        off, ref = ((t.double() - e).norm() / e.norm() for t in (a, b))
        # both round u, gelu(u), its gradient and every result to bf16 once (2^-9 each, 2^-8 with their sum): neither is further off
        assert off <= 2.0**-7 and off <= 1.05 * ref + 2.0**-14, (off, ref)
