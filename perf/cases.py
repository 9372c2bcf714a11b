"""The work whose time on one B200 is watched: what users of this library have it do, by family.

* ``train``: one data-parallel training step (``DataParallel`` + ``FlatAdamW`` in a ``GraphedTrainStep``);
* ``layer_norm``, ``xent``, ``adamw``: the layer, loss and optimizer entry points that people call from their
  own training loops, forward and backward;
* ``gemm``: ``gemm_bf16``, the product behind expert and tensor-parallel layers, from a few tokens (decode) to
  thousands (prefill, training);
* ``moe``: routing, dispatch and combine of an expert-parallel layer;
* ``allreduce``: the collective itself, small ordinary buffers and gradient buckets in the symmetric heap.

The two multi-rank families run with all ranks on the one GPU (``DeviceGroup.emulated``).
"""
import math

import torch

from oneccl_b200.models.gpt2 import GPT2, GPT2Config
from oneccl_b200.ops.device_group import DeviceGroup
from oneccl_b200.ops.gemm import gemm_bf16
from oneccl_b200.ops.nn import add_layer_norm
from oneccl_b200.ops.train import FlatAdamW, softmax_cross_entropy
from oneccl_b200.parallel.ddp import DataParallel, GraphedTrainStep
from oneccl_b200.parallel.ep import fused_combine, fused_dispatch, route_device

_DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16}
_PARAMS = {"gpt2-small": 124e6, "gpt2-medium": 354e6}


def listed():
    return [
        # the headline benchmark: GPT-2 medium, per-GPU batch 8 of 1024 tokens
        {"name": "train_medium_8x1024", "kind": "train", "model": "gpt2-medium", "batch": 8, "seq": 1024},
        # fine-tuning on a short ragged batch: many short kernels, the optimizer pass dominates the bytes
        {"name": "train_small_2x333", "kind": "train", "model": "gpt2-small", "batch": 2, "seq": 333},
        # residual add + LayerNorm, forward and backward, at the headline model's size
        {"name": "layer_norm_8192x1024", "kind": "layer_norm", "rows": 8192, "width": 1024},
        # the same for one short sequence at the width of the largest GPT-2
        {"name": "layer_norm_1023x1600", "kind": "layer_norm", "rows": 1023, "width": 1600},
        # the loss over the headline batch (vocabulary padded to 50304 columns)
        {"name": "xent_8192x50257", "kind": "xent", "rows": 8192, "vocab": 50257, "cols": 50304},
        # the loss of a small classifier or tokenizer, a ragged number of rows
        {"name": "xent_317x1000", "kind": "xent", "rows": 317, "vocab": 1000, "cols": 1024},
        # the optimizer step of GPT-2 small: clipping norm and AdamW over one flat buffer
        {"name": "adamw_124m", "kind": "adamw", "n": 124_475_904, "grad": "bfloat16"},
        # first product of an expert FFN on a training batch, SiLU in the epilogue
        {"name": "gemm_8192x14336x4096", "kind": "gemm", "m": 8192, "n": 14336, "k": 4096, "silu": True, "rows": 0},
        # the same expert while decoding: two dozen tokens, the weights are all that moves
        {"name": "gemm_24x14336x4096", "kind": "gemm", "m": 24, "n": 14336, "k": 4096, "silu": True, "rows": 0},
        # eight experts, top-2: route, dispatch to the experts, weighted combine
        {"name": "moe_8x1024x4096", "kind": "moe", "world": 8, "tokens": 1024, "hidden": 4096, "topk": 2},
        # a scalar-sized allreduce (loss, norm, counters) on ordinary buffers: latency only
        {"name": "allreduce_8x1027_fp32", "kind": "allreduce", "world": 8, "count": 1027, "dtype": "float32", "symm": False},
        # one 25 MiB gradient bucket in the symmetric heap, averaged in place
        {"name": "allreduce_8x25mib_bf16", "kind": "allreduce", "world": 8, "count": 13_107_200, "dtype": "bfloat16",
         "symm": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "layer_norm", "layer_norm", "xent", "xent", "adamw", "gemm", "gemm", "gemm", "moe",
                       "allreduce", "allreduce"])
    if kind == "train":
        model = rng.choice(["gpt2-small", "gpt2-medium"])
        return {"kind": kind, "model": model, "batch": rng.randint(1, 8), "seq": _log(rng, 64, 1024)}
    if kind == "layer_norm":
        return {"kind": kind, "rows": _log(rng, 64, 16384), "width": rng.choice([256, 512, 768, 1024, 1280, 1600])}
    if kind == "xent":
        vocab = _log(rng, 500, 50257)
        return {"kind": kind, "rows": _log(rng, 64, 8192), "vocab": vocab, "cols": (vocab + 63) // 64 * 64}
    if kind == "adamw":
        return {"kind": kind, "n": _log(rng, 100_000, 355_000_000), "grad": rng.choice(["bfloat16", "bfloat16", "float32"])}
    if kind == "gemm":
        m = _log(rng, 1, 8192)
        # every other one takes its row count from device memory, as the expert-parallel layer does
        rows = rng.randint(max(1, m // 8), m) if rng.random() < 0.5 else 0
        return {"kind": kind, "m": m, "n": 8 * _log(rng, 64, 1792), "k": 8 * _log(rng, 64, 1792), "silu": rng.random() < 0.5,
                "rows": rows}
    if kind == "moe":
        world = rng.choice([2, 4, 8])
        return {"kind": kind, "world": world, "tokens": _log(rng, 16, 2048), "hidden": 8 * _log(rng, 64, 512),
                "topk": rng.choice([1, 2, 2])}
    if rng.random() < 0.5:
        return {"kind": kind, "world": rng.choice([2, 4, 8]), "count": _log(rng, 1, 65536), "dtype": rng.choice(list(_DTYPES)),
                "symm": False}
    return {"kind": kind, "world": rng.choice([2, 4, 8]), "count": 8 * _log(rng, 65536, 3_000_000),
            "dtype": rng.choice(["float32", "bfloat16"]), "symm": True}


def prepare(case, seed):
    return _FAMILY[case["kind"]][0](case, torch.Generator(device="cuda").manual_seed(seed))


def run(state):
    return state["run"](state)


def work(case):
    return _FAMILY[case["kind"]][1](case)


def tolerance(case):
    return _FAMILY[case["kind"]][2](case)


def _randn(g, *shape, dtype=torch.bfloat16):
    return torch.randn(*shape, generator=g, device="cuda").to(dtype)


# ---- training step ------------------------------------------------------------------------------------

def _train_prepare(case, g):
    base = GPT2Config.named(case["model"])
    cfg = GPT2Config(base.n_layer, base.n_head, base.d_model, case["seq"], base.vocab)
    torch.manual_seed(g.initial_seed())
    with torch.device("cuda"):
        model = GPT2(cfg).to(torch.bfloat16)
    group = DeviceGroup.emulated(1, heap_bytes=1 << 30, staging_bytes=16 << 20)
    ddp = DataParallel(model, group)
    opt = ddp.make_optimizer(device_step=True)
    idx, tgt = (torch.randint(0, cfg.vocab, (case["batch"], case["seq"]), generator=g, device="cuda") for _ in range(2))
    return {"run": _train_run, "step": GraphedTrainStep(ddp, opt, idx, tgt), "idx": idx, "tgt": tgt, "group": group}


def _train_run(s):
    step = s["step"]
    loss = step(s["idx"], s["tgt"])
    ddp, opt = step.ddp, step.opt
    return loss, ddp.flat_grad, ddp.flat_param, opt.master, opt.m, opt.v


def _train_work(case):
    base = GPT2Config.named(case["model"])
    n, tokens = _PARAMS[case["model"]], case["batch"] * case["seq"]
    # 6 flops per parameter and token, and causal attention: 2 products forward, 5 backward
    attention = 7 * tokens * case["seq"] * base.d_model * base.n_layer
    # optimizer: gradient read, master, m and v read and written, bf16 parameters written; parameters read once
    return {"bytes": n * (2 + 24 + 2 + 2), "flops": 6 * n * tokens + attention}


def _train_tolerance(case):
    # bf16 activations and gradients; the first AdamW steps turn a tiny gradient's sign into a whole step
    return {"rel": 2e-2, "max": 0.5}


# ---- LayerNorm with the residual addition ----------------------------------------------------------------

def _ln_prepare(case, g):
    rows, width = case["rows"], case["width"]
    ins = [_randn(g, rows, width), _randn(g, rows, width), 1 + 0.1 * _randn(g, width), 0.1 * _randn(g, width)]
    return {"run": _ln_run, "ins": [t.requires_grad_(True) for t in ins],
            "grads": [_randn(g, rows, width), _randn(g, rows, width)]}


def _ln_run(s):
    y, total = add_layer_norm(*s["ins"])
    return (y.detach(), total.detach(), *torch.autograd.grad([y, total], s["ins"], s["grads"]))


def _ln_work(case):
    n = case["rows"] * case["width"]
    # forward: x, residual -> y, sum; backward: dy, dsum, sum -> dx (the residual's gradient is the same tensor)
    return {"bytes": 2 * n * (4 + 4), "flops": 20 * n}


def _bf16_tolerance(case):
    return {"rel": 1e-2}


# ---- cross-entropy ------------------------------------------------------------------------------------------

def _xent_prepare(case, g):
    logits = _randn(g, case["rows"], case["cols"]).mul_(2.5).requires_grad_(True)
    targets = torch.randint(0, case["vocab"], (case["rows"],), generator=g, device="cuda")
    return {"run": _xent_run, "logits": logits, "targets": targets, "vocab": case["vocab"]}


def _xent_run(s):
    # the logits are consumed: they hold their gradient afterwards, and a further pass reads that as logits
    loss = softmax_cross_entropy(s["logits"], s["targets"], s["vocab"])
    (grad,) = torch.autograd.grad(loss, s["logits"])
    return loss.detach(), grad


def _xent_work(case):
    n = case["rows"] * case["cols"]
    return {"bytes": 4 * n + 8 * case["rows"], "flops": 6 * n}


# ---- optimizer ------------------------------------------------------------------------------------------------

def _adamw_prepare(case, g):
    n = case["n"]
    opt = FlatAdamW(_randn(g, n).mul_(0.02), n // 8 * 7)
    return {"run": _adamw_run, "opt": opt, "grad": _randn(g, n, dtype=_DTYPES[case["grad"]]).mul_(1e-3)}


def _adamw_run(s):
    opt = s["opt"]
    opt.step(s["grad"])
    return opt.model_flat, opt.master, opt.m, opt.v, opt.grad_norm()


def _adamw_work(case):
    g = 2 if case["grad"] == "bfloat16" else 4
    # the gradient is read for the norm and, unless it fits on the chip, again for the update
    return {"bytes": case["n"] * ((1 if case["n"] * g < 100e6 else 2) * g + 24 + 2), "flops": 18 * case["n"]}


def _adamw_tolerance(case):
    return {"rel": 1e-4, "max": 1e-2}  # the bf16 copy may round the other way


# ---- bf16 product -------------------------------------------------------------------------------------------------

def _gemm_prepare(case, g):
    m, n, k = case["m"], case["n"], case["k"]
    rows = torch.tensor([case["rows"]], dtype=torch.int32, device="cuda") if case["rows"] else None
    return {"run": _gemm_run, "a": _randn(g, m, k), "w": _randn(g, n, k).mul_(0.02), "rows": rows,
            "out": torch.zeros(m, n, dtype=torch.bfloat16, device="cuda"), "epilogue": "silu" if case["silu"] else None}


def _gemm_run(s):
    return gemm_bf16(s["a"], s["w"], out=s["out"], epilogue=s["epilogue"], rows=s["rows"])


def _gemm_work(case):
    m = case["rows"] or case["m"]
    return {"bytes": 2 * (m * case["k"] + case["n"] * case["k"] + m * case["n"]), "flops": 2 * m * case["n"] * case["k"]}


# ---- expert-parallel exchange ----------------------------------------------------------------------------------------

def _moe_prepare(case, g):
    W, T, H, k = case["world"], case["tokens"], case["hidden"], case["topk"]
    cap = T * k * W
    group = DeviceGroup.emulated(W, heap_bytes=cap * H * 2 + (24 << 20), staging_bytes=4 << 20)
    xs = [_randn(g, T, H) for _ in range(W)]
    return {"run": _moe_run, "group": group, "topk": k, "x": xs,
            "logits": [torch.randn(T, W, generator=g, device="cuda") for _ in range(W)],
            "recv": group.symm_empty((cap, H), dtype=torch.bfloat16),
            "counts": group.symm_empty((256 * W * W,), dtype=torch.int32),
            "meta": [torch.zeros(2 * W + 2, dtype=torch.int32, device="cuda") for _ in range(W)],
            "out": [torch.empty_like(x) for x in xs]}


def _moe_run(s):
    k = s["topk"]
    idx, wts, counts, order, pos = zip(*(route_device(lg, k) for lg in s["logits"]))
    fused_dispatch(s["group"], s["x"], order, counts, s["meta"], s["recv"], s["counts"], k)
    # the experts' products are the gemm family: here the rows come back as they arrived
    fused_combine(s["group"], [i.view(-1) for i in idx], pos, [w.view(-1) for w in wts], s["out"], s["meta"], s["recv"], k)
    return list(s["out"]), list(s["meta"]), idx, wts


def _moe_work(case):
    W, T, H, k = case["world"], case["tokens"], case["hidden"], case["topk"]
    rows = W * T * H * 2
    # dispatch: x -> k copies of every row; combine: k rows -> one; routing: logits -> ids and weights
    return {"bytes": rows * (1 + k + k + 1) + W * T * (4 * W + 12 * k), "flops": W * T * H * k * 2}


# ---- allreduce ------------------------------------------------------------------------------------------------------------

def _allreduce_prepare(case, g):
    W, n, dtype = case["world"], case["count"], _DTYPES[case["dtype"]]
    size = n * torch.empty((), dtype=dtype).element_size()
    if case["symm"]:
        group = DeviceGroup.emulated(W, heap_bytes=size + (16 << 20), staging_bytes=1 << 20)
        send = recv = group.symm_empty((n,), dtype=dtype)
        for t in send:
            t.copy_(_randn(g, n, dtype=dtype))
    else:
        group = DeviceGroup.emulated(W, heap_bytes=4 << 20)
        send = [_randn(g, n, dtype=dtype) for _ in range(W)]
        recv = [torch.empty_like(t) for t in send]
    return {"run": _allreduce_run, "group": group, "send": send, "recv": recv, "scale": 1.0 / W if case["symm"] else None}


def _allreduce_run(s):
    return s["group"].allreduce(s["send"], s["recv"], scale=s["scale"])


def _allreduce_work(case):
    size = case["count"] * torch.empty((), dtype=_DTYPES[case["dtype"]]).element_size()
    return {"bytes": 2 * case["world"] * size, "flops": case["world"] * case["count"]}


def _allreduce_tolerance(case):
    return {"rel": 1e-5 if case["dtype"] == "float32" else 1e-2 if case["dtype"] == "bfloat16" else 1e-3}


_FAMILY = {
    "train": (_train_prepare, _train_work, _train_tolerance),
    "layer_norm": (_ln_prepare, _ln_work, _bf16_tolerance),
    "xent": (_xent_prepare, _xent_work, _bf16_tolerance),
    "adamw": (_adamw_prepare, _adamw_work, _adamw_tolerance),
    "gemm": (_gemm_prepare, _gemm_work, _bf16_tolerance),
    "moe": (_moe_prepare, _moe_work, _bf16_tolerance),
    "allreduce": (_allreduce_prepare, _allreduce_work, _allreduce_tolerance),
}
