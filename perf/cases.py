"""Workloads of the optimizer-step path for timing, through the package's public calls.

A case is a dict of plain values.  ``call`` names the entry point:

  op_sgd      raf_b200.op.sgd, the operator that returns new tensors
  eager_sgd   raf_b200.optim.SGD.step over the parameters of a small network
  eager_lans  raf_b200.optim.LANS.step (one raf.op.lans call over every parameter)
  with_lans   the ZeRO-aware wrapper raf_b200.optim.with_lans on a 16-bit model
  zero        raf_b200.zero.ZeroStep.step: the bound step a training loop repeats
  host        raf_b200.zero.ZeroStep.step_host: pinned gradients in, parameters out
  group_cast  raf_b200.op.group_cast: a list of gradients to another type
  bucket      raf_b200.op.fuse_tensor, then defuse_tensor: a bucket packed and unpacked

The tensors of a case come from ``net``: a BERT- or GPT-2-shaped transformer (with ``ranks`` > 1
the row blocks that rank 0 of that many owns), a bottleneck ResNet, one flat tensor, or a list of
ragged sizes.
"""
import math
import random

import numpy as np
import torch

from raf_b200 import distributed as dist
from raf_b200 import op, optim
from raf_b200.zero import Plan, ZeroStep, make_hyper

_DT = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}
_BYTES = {"float32": 4, "float16": 2, "bfloat16": 2}
_LARGEST = 335_141_888 * 28  # bytes of one LANS step over the BERT-large list, the largest case


# ---- shapes --------------------------------------------------------------------------------------
def _bert(layers, hidden, vocab, positions):
    ffn = 4 * hidden
    s = [(vocab, hidden), (positions, hidden), (2, hidden), (hidden,), (hidden,)]
    for _ in range(layers):
        s += _encoder_layer(hidden, ffn)
    return s + [(hidden, hidden), (hidden,)]


def _encoder_layer(hidden, ffn):
    s = []
    for _ in range(4):
        s += [(hidden, hidden), (hidden,)]
    s += [(hidden,), (hidden,)]
    s += [(ffn, hidden), (ffn,), (hidden, ffn), (hidden,)]
    return s + [(hidden,), (hidden,)]


def _gpt2(layers, d, vocab, positions):
    s = [(vocab, d), (positions, d)]
    for _ in range(layers):
        s += [(d,), (d,), (d, 3 * d), (3 * d,), (d, d), (d,)]
        s += [(d,), (d,), (d, 4 * d), (4 * d,), (4 * d, d), (d,)]
    return s + [(d,), (d,)]


def _resnet(width, blocks, classes):
    s = []

    def conv_bn(o, i, k):
        s.extend([(o, i, k, k), (o,), (o,)])

    conv_bn(width, 3, 7)
    inplanes = width
    for stage, n in enumerate(blocks):
        planes = width << stage
        for b in range(n):
            conv_bn(planes, inplanes, 1)
            conv_bn(planes, planes, 3)
            conv_bn(planes * 4, planes, 1)
            if b == 0:
                conv_bn(planes * 4, inplanes, 1)
            inplanes = planes * 4
    return s + [(classes, inplanes), (classes,)]


def _ragged(count, low, high, pick):
    """`count` one-dimensional tensors, sizes log-uniform in [low, high], whatever they divide by."""
    r = random.Random(pick)
    return [(int(round(math.exp(r.uniform(math.log(low), math.log(high))))),) for _ in range(count)]


def _numel(shape):
    n = 1
    for d in shape:
        n *= d
    return n


def _shapes(c):
    net = c["net"]
    if net == "bert":
        s = _bert(c["layers"], c["hidden"], c["vocab"], c["positions"])
    elif net == "gpt2":
        s = _gpt2(c["layers"], c["hidden"], c["vocab"], c["positions"])
    elif net == "encoder":
        s = [x for _ in range(c["layers"]) for x in _encoder_layer(c["hidden"], 4 * c["hidden"])]
    elif net == "resnet":
        s = _resnet(c["width"], [int(ch) for ch in str(c["blocks"])], c["classes"])
    elif net == "flat":
        s = [(c["elements"],)]
    elif net == "small":  # a convolution and a classifier, a few thousand elements
        s = [(c["width"], 3, 3, 3), (c["width"],), (10, c["width"]), (10,), (7, 5)]
    else:
        s = _ragged(c["count"], c["low"], c["high"], c["pick"])
    ranks = c.get("ranks", 1)
    if ranks > 1:  # rows are split, the last block padded
        s = [(-(-x[0] // ranks),) + x[1:] for x in s]
    return s


# ---- the cases -----------------------------------------------------------------------------------
def listed():
    return [
        # One convolution weight through the operator itself: what a call costs at least.
        {"name": "op_sgd_conv64", "call": "op_sgd", "net": "flat", "elements": 1728, "grad": "float32"},
        # The eager loop over a small ResNet (one bottleneck block a stage, 53 tensors): a launch per parameter.
        {"name": "eager_sgd_resnet53", "call": "eager_sgd", "net": "resnet", "width": 64, "blocks": 1111,
         "classes": 1000, "momentum": 0.9},
        # The eager LANS optimizer on a network of a few thousand parameters.
        {"name": "eager_lans_small", "call": "eager_lans", "net": "small", "width": 64},
        # The ZeRO-aware wrapper around one encoder layer with fp16 parameters and gradients.
        {"name": "with_lans_layer_f16", "call": "with_lans", "net": "encoder", "layers": 1, "hidden": 1024,
         "grad": "float16", "param": "float16"},
        # SGD with momentum and weight decay on ResNet-50, all fp32 (161 tensors).
        {"name": "zero_sgd_resnet50", "call": "zero", "optimizer": "sgd", "net": "resnet", "width": 64, "blocks": 3463,
         "classes": 1000, "grad": "float32", "param": "float32"},
        # What each of eight ranks updates of BERT-large with LANS, fp16 gradients under a loss scale.
        {"name": "zero_lans_bert_shard8", "call": "zero", "optimizer": "lans", "net": "bert", "layers": 24,
         "hidden": 1024, "vocab": 30522, "positions": 512, "ranks": 8, "grad": "float16", "param": "float16"},
        # All of BERT-large on one GPU: the largest step.
        {"name": "zero_lans_bert", "call": "zero", "optimizer": "lans", "net": "bert", "layers": 24, "hidden": 1024,
         "vocab": 30522, "positions": 512, "ranks": 1, "grad": "float16", "param": "float16"},
        # What each of eight ranks updates of GPT-2-medium with Adam, bf16 gradients and copies.
        {"name": "zero_adam_gpt2_shard8", "call": "zero", "optimizer": "adam", "net": "gpt2", "layers": 24,
         "hidden": 1024, "vocab": 50257, "positions": 1024, "ranks": 8, "grad": "bfloat16", "param": "bfloat16"},
        # One flat fp32 tensor, Adam, out of the middle of the bucket-size sweep.
        {"name": "zero_adam_flat16m", "call": "zero", "optimizer": "adam", "net": "flat", "elements": 16 << 20,
         "grad": "float32", "param": "float32"},
        # End to end from host memory: ResNet-50 gradients in, parameters back.
        {"name": "host_sgd_resnet50", "call": "host", "optimizer": "sgd", "net": "resnet", "width": 64, "blocks": 3463,
         "classes": 1000, "grad": "float32", "param": "float32"},
        # The fp16 gradients of two encoder layers to fp32, as in front of an fp32-only update.
        {"name": "group_cast_2layers", "call": "group_cast", "net": "encoder", "layers": 2, "hidden": 1024,
         "grad": "float16", "to": "float32"},
        # A gradient bucket of odd sizes packed into one buffer and taken apart again.
        {"name": "bucket_ragged48", "call": "bucket", "net": "ragged", "count": 48, "low": 200, "high": 1 << 20,
         "pick": 7, "grad": "float32"},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    while True:
        c = _draw(rng)
        if work(c)["bytes"] <= _LARGEST:
            return c


def _draw(rng):
    f = rng.choice(["float32", "float16", "bfloat16"])
    call = rng.choice(["op_sgd", "eager_sgd", "eager_lans", "with_lans", "zero", "zero", "zero", "zero", "host",
                       "group_cast", "bucket"])
    if call == "op_sgd":
        return {"call": call, "net": "flat", "elements": _log(rng, 1, 4 << 20), "grad": f}
    if call == "eager_sgd":
        return {"call": call, "net": "resnet", "width": rng.randint(5, 64),
                "blocks": rng.choice([1111, 111, 11, 21]), "classes": rng.randint(2, 1000),
                "momentum": rng.choice([0.0, 0.9])}
    if call == "eager_lans":
        if rng.random() < 0.5:
            return {"call": call, "net": "small", "width": rng.randint(3, 600)}
        return {"call": call, "net": "ragged", "count": rng.randint(1, 31), "low": 10, "high": _log(rng, 100, 4 << 20),
                "pick": rng.randrange(1 << 30)}
    if call == "with_lans":
        return {"call": call, "net": "encoder", "layers": 1, "hidden": rng.randint(33, 1280), "grad": f, "param": f}
    if call == "group_cast":
        return {"call": call, "net": "encoder", "layers": rng.randint(1, 4), "hidden": rng.randint(33, 1280),
                "grad": f, "to": rng.choice([t for t in ("float32", "float16", "bfloat16") if t != f])}
    if call == "bucket":
        return {"call": call, "net": "ragged", "count": rng.randint(1, 60), "low": 10, "high": _log(rng, 1000, 8 << 20),
                "pick": rng.randrange(1 << 30), "grad": f}
    c = {"call": call, "optimizer": rng.choice(["sgd", "adam", "lans"])}
    net = rng.choice(["bert", "gpt2", "resnet", "flat", "ragged"])
    c["net"] = net
    if net in ("bert", "gpt2"):
        hidden = rng.choice([8 * rng.randint(8, 160), rng.randint(64, 1280)])
        c.update(layers=rng.randint(1, 24), hidden=hidden, vocab=_log(rng, 1000, 60000),
                 positions=rng.choice([128, 512, 1024]), ranks=rng.choice([1, 2, 4, 8]))
    elif net == "resnet":
        c.update(width=rng.randint(8, 80), blocks=rng.choice([3463, 2222, 1111]), classes=rng.randint(2, 1000),
                 ranks=rng.choice([1, 2, 4, 8]))
    elif net == "flat":
        c.update(elements=_log(rng, 1000, 256 << 20))
    else:
        c.update(count=rng.randint(2, 300), low=1, high=_log(rng, 1000, 4 << 20), pick=rng.randrange(1 << 30))
    if call == "host" and sum(map(_numel, _shapes(c))) > 64 << 20:
        return _draw(rng)  # the copies over PCIe take tens of milliseconds from there on
    c["grad"] = f
    c["param"] = f if rng.random() < 0.8 else "float32"
    if c["optimizer"] == "lans" and rng.random() < 0.15:
        c["normalize"] = False
    return c


# ---- what a program has in hand before the call --------------------------------------------------
def _arena(sizes, dtype, host=False):
    """One allocation and, for every tensor, the view at the next multiple of 256 bytes, where an
    allocator would put it."""
    es = torch.empty((), dtype=dtype).element_size()
    per, at, offs = 256 // es, 0, []
    for n in sizes:
        offs.append(at)
        at += -(-n // per) * per
    buf = torch.zeros(at, dtype=dtype, pin_memory=True) if host else torch.zeros(at, dtype=dtype, device="cuda")
    return buf, [buf[o:o + n] for o, n in zip(offs, sizes)]


def _fill(views, std, gen):
    for x in views:
        x.copy_(torch.randn(x.numel(), generator=gen, device="cuda") * std)


def prepare(case, seed):
    c = dict(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    shapes = _shapes(c)
    sizes = [_numel(s) for s in shapes]
    s = {"case": c, "step": 0}
    gdt = _DT[c.get("grad", "float32")]
    # fp16 gradients carry a loss scale of 2^15, as in mixed-precision training
    scale = 2.0 ** 15 if gdt == torch.float16 else 1.0
    call = c["call"]
    if call in ("group_cast", "bucket"):
        _, views = _arena(sizes, gdt)
        _fill(views, 1e-3 * scale, gen)
        s["tensors"] = [x.view(sh) for x, sh in zip(views, shapes)]
        if call == "bucket":
            s["sizes"] = sizes
            s["dims"] = [d for sh in shapes for d in sh]
            s["ends"] = [int(x) for x in np.cumsum([len(sh) for sh in shapes])]
        return s
    if call == "op_sgd":
        n = sizes[0]
        s["x"] = torch.randn(n, generator=gen, device="cuda") * 0.02
        s["v"] = torch.randn(n, generator=gen, device="cuda") * 1e-3
        s["dx"] = (torch.randn(n, generator=gen, device="cuda") * 1e-3).to(gdt)
        return s
    gbuf, grads = _arena(sizes, gdt)
    _fill(grads, 1e-3 * scale, gen)
    if call in ("eager_sgd", "eager_lans", "with_lans"):
        pdt = _DT[c.get("param", "float32")]
        s["pbuf"], params = _arena(sizes, pdt)
        _fill(params, 0.02, gen)
        params = [x.view(sh) for x, sh in zip(params, shapes)]
        s["grads"] = [g.view(sh) for g, sh in zip(grads, shapes)]
        if call == "with_lans":
            model = {"layer.%d" % i: p for i, p in enumerate(params)}
            s["opt"] = optim.with_lans(lr=1e-3)(model, grad_dtype=gdt, grad_scale=1.0 / scale)
            return s
        for p, g in zip(params, s["grads"]):
            p.grad = g
        s["opt"] = optim.SGD(params, 0.1, c["momentum"]) if call == "eager_sgd" else optim.LANS(params)
        return s
    # the bound step: fp32 master, first and second moment in the middle of training, gradients and
    # the model's own parameters
    pdt = _DT[c["param"]]
    which = c["optimizer"]
    s["p"], p = _arena(sizes, torch.float32)
    s["m"], m = _arena(sizes, torch.float32)
    _fill(p, 0.02, gen)
    _fill(m, 3e-4, gen)
    v = None
    if which != "sgd":
        s["v"], v = _arena(sizes, torch.float32)
        for x in v:
            x.copy_(1e-6 * (0.5 + torch.rand(x.numel(), generator=gen, device="cuda")))
    pbuf, params = s["p"], p  # an fp32 model on one rank is its own master copy
    if pdt != torch.float32:
        pbuf, params = _arena(sizes, pdt)
    s["out"] = pbuf
    s["plan"] = Plan([(n,) for n in sizes], 1, 0, 13107200)
    s["zero"] = ZeroStep(s["plan"], dist.get_communicator(), gdt, pdt, which)
    s["zero"].bind(grads, params, p, m, v)
    if which == "sgd":
        s["hyper"] = make_hyper("sgd", learning_rate=0.1, mu=0.9, weight_decay=1e-4, grad_scale=1.0 / scale)
    elif which == "adam":
        s["hyper"] = make_hyper("adam", learning_rate=1e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1,
                                grad_scale=1.0 / scale)
    else:
        s["hyper"] = make_hyper("lans", learning_rate=1e-3, beta1=0.9, beta2=0.999, eps=1e-6, weight_decay=0.01,
                                normalize_grad=int(c.get("normalize", True)), grad_scale=1.0 / scale)
    s["step"] = 100
    if call == "host":
        hg, s["grads_host"] = _arena(sizes, gdt, host=True)
        s["host_out"], s["params_host"] = _arena(sizes, pdt, host=True)
        for a, b in zip(s["grads_host"], grads):
            a.copy_(b)
        gbuf.zero_()
        for one in (hg, s["host_out"], gbuf, pbuf):
            s["zero"].declare_arena(one)
    return s


# ---- one pass ------------------------------------------------------------------------------------
def run(s):
    c = s["case"]
    call = c["call"]
    if call == "op_sgd":
        return op.sgd(s["x"], s["dx"], s["v"], 0.1, 0.9)
    if call == "group_cast":
        return op.group_cast(s["tensors"], c["to"])
    if call == "bucket":
        flat = op.fuse_tensor(s["tensors"])
        return flat, op.defuse_tensor(flat, s["sizes"], s["dims"], s["ends"])
    if call in ("eager_sgd", "eager_lans"):
        s["opt"].step()
        return s["pbuf"], s["opt"].state()
    if call == "with_lans":
        s["opt"].step(s["grads"])
        return s["pbuf"], s["opt"].state
    s["step"] += 1
    if call == "host":
        s["zero"].step_host(s["hyper"], s["step"], s["grads_host"], s["params_host"])
        return s["host_out"], s["p"], s["m"], s.get("v")
    s["zero"].step(s["hyper"], s["step"])
    return s["out"], s["p"], s["m"], s.get("v")


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    n = sum(_numel(x) for x in _shapes(case))
    g = _BYTES[case.get("grad", "float32")]
    call = case["call"]
    if call == "group_cast":
        return {"bytes": n * (g + _BYTES[case["to"]]), "flops": 0}
    if call == "bucket":  # read and written once each way
        return {"bytes": n * g * 4, "flops": 0}
    if call in ("op_sgd", "eager_sgd"):
        return {"bytes": n * (g + 4 + 4 + 8), "flops": 4 * n}
    which = case.get("optimizer", "lans")
    state = 8 if which == "sgd" else 12  # p, m (and v), read and written
    out = _BYTES[case.get("param", "float32")]
    out = 0 if out == 4 else out  # an fp32 model is its own master copy
    if call == "with_lans":
        out = _BYTES[case["param"]]  # the wrapper keeps a master copy of its own
    return {"bytes": n * (g + 2 * state + out), "flops": n * {"sgd": 6, "adam": 14, "lans": 32}[which]}


def tolerance(case):
    """Casts and copies are whole; SGD and Adam round each fp32 operation (1e-6); the norms of LANS
    are fp32 sums over a tensor (1e-5).  Where a 16-bit copy of the parameters comes back, a master
    value next to a rounding boundary may land on the other side: one unit of that type at most,
    and that on few elements."""
    if case["call"] in ("group_cast", "bucket"):
        return "exact"
    lans = case.get("optimizer", "lans") == "lans" and case["call"] not in ("op_sgd", "eager_sgd")
    rel = 1e-5 if lans else 1e-6
    out = case.get("param", "float32")
    if out == "float32":
        return {"rel": rel, "max": 40 * rel}
    ulp = 2.0 ** -10 if out == "float16" else 2.0 ** -7
    # a share of about rel / ulp of the values crosses a boundary, each by at most one unit
    return {"rel": math.sqrt(rel / ulp) * ulp, "max": ulp}
