"""Work that programs built on this package have it do on one GPU, as cases that can be timed.

A case is a dict of plain values. `listed()` are the standing ones, `draw(rng)` gives others of the same ranges,
`prepare(case, seed)` makes what a program holds before the call, `run(state)` is one pass through the public entry
points, `work(case)` the bytes and operations that such a pass cannot do without, and `tolerance(case)` how far
the outputs of two correct implementations may lie apart.

    allreduce    the named API on an ordinary tensor (a group of one rank)
    emu_*        the collective kernels among 2 to 8 ranks emulated on one GPU, grid sizes as in bench/kernel_cases.py
    optimizer    `DistributedOptimizer.step()` with the update fused behind the reduction, gradients brought by the caller
    gru_*        `nn.GRU` stacks on the persistent kernels: outputs only (inference), or outputs and all gradients
    bn_clip      batch norm with the clipped ReLU, forward and backward
    ds2_step     a whole training step of the speech model: zero_grad, loss, backward, step
"""
from __future__ import annotations

import math
import os
import random

import torch

import tensorflow_allreduce_b200 as bc
from tensorflow_allreduce_b200.models import ds2, gpt2, resnet50
from tensorflow_allreduce_b200.ops import persistent_gru
from tensorflow_allreduce_b200.ops.bn_clip import BatchNormClip2d
from tensorflow_allreduce_b200.ops.emulated import EmulatedGroup

_DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16, "int32": torch.int32, "int64": torch.int64}
_SIZES = {"fp32": 4, "bf16": 2, "fp16": 2, "int32": 4, "int64": 8}
_CLIP = 20.0


def listed():
    return [
        # A metric or a small gradient averaged by name every step: the [1000, 10] tensor of the plumbing configuration.
        {"name": "allreduce_10k_fp32", "kind": "allreduce", "dtype": "fp32", "numel": 10000, "average": True},
        # A large ordinary tensor (not in symmetric memory), an element count that no vector width divides.
        {"name": "allreduce_256MiB_bf16", "kind": "allreduce", "dtype": "bf16", "numel": (128 << 20) + 13, "average": False},
        # Small per-layer gradients among 8 ranks, one-shot, the largest message that path takes by default.
        {"name": "emu8_one_shot_256KiB", "kind": "emu_one_shot", "dtype": "fp32", "ranks": 8, "numel": 64 << 10},
        # A large gradient bucket among 8 ranks, reduced in place.
        {"name": "emu8_two_shot_64MiB", "kind": "emu_two_shot", "dtype": "fp32", "ranks": 8, "numel": 16 << 20},
        # Sparse gradients: rank r brings (r + 1) * rows rows of 256.
        {"name": "emu8_allgatherv_rows", "kind": "emu_allgatherv", "dtype": "fp32", "ranks": 8, "rows": 911, "width": 256},
        # The update of ResNet-50 (many small tensors), momentum-SGD on bf16 gradients with fp32 master weights.
        {"name": "sgd_resnet50_bf16", "kind": "optimizer", "model": "resnet50", "classes": 1000},
        # The update of GPT-2 medium: AdamW on bf16 gradients with fp32 master weights.
        {"name": "adamw_gpt2_medium_bf16", "kind": "optimizer", "model": "gpt2", "layers": 24, "width": 1024, "vocab": 50257},
        # Recognising a few short utterances: a stack of GRU layers without gradients.
        {"name": "gru_infer_T75_B3_H512", "kind": "gru_infer", "T": 75, "B": 3, "I": 200, "H": 512, "layers": 2, "dirs": 2},
        # One recurrent layer of the speech model in training.
        {"name": "gru_train_T350_B32_H1024", "kind": "gru_train", "T": 350, "B": 32, "I": 2048, "H": 1024, "layers": 1, "dirs": 2},
        # The norms of the speech model: the full-size first block, and the second block for a short, odd batch.
        {"name": "bn_clip_32x32x81x350", "kind": "bn_clip", "N": 32, "C": 32, "H": 81, "W": 350},
        {"name": "bn_clip_5x32x41x175", "kind": "bn_clip", "N": 5, "C": 32, "H": 41, "W": 175},
        # The headline configuration: a whole training step, batch 32 of 161 x 700 spectrograms.
        {"name": "ds2_step_b32", "kind": "ds2_step", "batch": 32, "frames": 700, "hidden": 1024, "layers": 5, "labels": 100},
    ]


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["allreduce", "allreduce", "emu_one_shot", "emu_two_shot", "emu_allgatherv", "optimizer", "optimizer", "gru_infer",
                       "gru_infer", "gru_train", "gru_train", "bn_clip", "bn_clip", "ds2_step"])
    c = {"kind": kind}
    if kind == "allreduce":
        c["dtype"] = rng.choice(sorted(_DTYPES))
        c["numel"] = max(1, _log(rng, 17 * 4, 512 << 20) // _SIZES[c["dtype"]])
        c["average"] = rng.random() < 0.5
    elif kind == "emu_one_shot":
        c["dtype"] = rng.choice(["fp32", "bf16", "fp16"])
        c["ranks"] = rng.choice([2, 4, 8])
        c["numel"] = _log(rng, 4 << 10, 256 << 10) // _SIZES[c["dtype"]]
    elif kind == "emu_two_shot":
        c["dtype"] = rng.choice(["fp32", "bf16", "fp16"])
        c["ranks"] = rng.choice([2, 4, 8])
        c["numel"] = _log(rng, 1 << 20, 128 << 20) // _SIZES[c["dtype"]]
    elif kind == "emu_allgatherv":
        c["dtype"] = rng.choice(["fp32", "bf16"])
        c["ranks"] = rng.choice([2, 4, 8])
        c["rows"] = _log(rng, 10, 2000)
        c["width"] = rng.choice([4, 64, 255, 256, 1024])
    elif kind == "optimizer":
        c["model"] = rng.choice(["resnet50", "gpt2", "ds2"])
        if c["model"] == "resnet50":
            c["classes"] = _log(rng, 10, 20000)
        elif c["model"] == "gpt2":
            c["layers"] = rng.randint(1, 24)
            c["width"] = rng.choice([256, 512, 768, 1024])
            c["vocab"] = _log(rng, 1000, 50257)
        else:
            c["layers"] = rng.randint(1, 5)
            c["hidden"] = 128 * rng.randint(1, 8)
    elif kind in ("gru_infer", "gru_train"):
        c["T"] = _log(rng, 12, 700 if kind == "gru_infer" else 350)
        c["B"] = rng.randint(1, 32)
        c["H"] = 128 * rng.randint(1, 8)
        c["I"] = rng.choice([40, 200, 1312, 2 * c["H"]])
        c["layers"] = rng.randint(1, 5 if kind == "gru_infer" else 2)
        c["dirs"] = rng.choice([1, 2, 2])
    elif kind == "bn_clip":
        c["N"] = rng.randint(2, 32)
        c["C"] = rng.choice([8, 16, 32, 32, 32])
        c["H"] = rng.choice([13, 41, 81])
        c["W"] = _log(rng, 17, 350)
    else:
        c["batch"] = rng.randint(4, 32)
        c["frames"] = rng.randint(100, 700)
        c["hidden"] = 128 * rng.randint(1, 8)
        c["layers"] = rng.randint(1, 5)
        c["labels"] = max(5, c["frames"] // 8)
    return c


def _join_group():
    """The group of one rank that a program on one GPU forms, and the math modes of the benchmark configurations."""
    torch.backends.cudnn.allow_tf32 = True
    torch.backends.cuda.matmul.allow_tf32 = True
    if not bc.is_initialized():
        for k in ("RANK", "WORLD_SIZE", "LOCAL_RANK"):
            os.environ.pop(k, None)
        bc.init(device=0)


def _values(gen, numel, dtype):
    if dtype in (torch.int32, torch.int64):
        return torch.randint(-100000, 100000, (numel,), dtype=dtype, device="cuda", generator=gen)
    return (torch.rand(numel, device="cuda", generator=gen) * 2 - 1).to(dtype)      # U(-1, 1), as in the bandwidth sweep


def _buffers(group, dtype, numel):
    """Views of every rank's buffer, each of which keeps the group (the owner of that memory) alive."""
    views = [group.buffer(r, dtype, numel) for r in range(group.nranks)]
    for v in views:
        v.owner = group
    return views


def _whole_storages(tensors):
    """One flat tensor over each storage that `tensors` live in."""
    out, seen = [], set()
    for t in tensors:
        s = t.untyped_storage()
        if s.data_ptr() not in seen:
            seen.add(s.data_ptr())
            out.append(torch.empty(0, dtype=t.dtype, device=t.device).set_(s, 0, (s.nbytes() // t.element_size(),)))
    return out


def _wrap(model, base, gen):
    """`DistributedOptimizer` around an optimizer that has run before: its state holds values. Also the flat views of the
    parameters and of the state."""
    params = [p for g in base.param_groups for p in g["params"]]
    sgd = isinstance(base, torch.optim.SGD)
    if sgd:
        for p in params:
            base.state[p]["momentum_buffer"] = torch.zeros_like(p, dtype=torch.float32)
    opt = bc.DistributedOptimizer(base)
    flats = _whole_storages(params)
    for key in ("momentum_buffer",) if sgd else ("exp_avg", "exp_avg_sq"):
        for s in _whole_storages([opt.state[p][key] for p in params]):
            s.normal_(generator=gen).mul_(1e-3)
            if key == "exp_avg_sq":
                s.square_()
            flats.append(s)
    return opt, params, flats


def _optimizer_model(case):
    with torch.device("cuda"):
        if case["model"] == "resnet50":
            model = resnet50.ResNet50(case["classes"]).to(torch.bfloat16).to(memory_format=torch.channels_last)
            return model, torch.optim.SGD(model.parameters(), lr=0.1, momentum=0.9, weight_decay=1e-4)
        if case["model"] == "gpt2":
            w = case["width"]
            model = gpt2.GPT2(gpt2.GPT2Config(n_layer=case["layers"], d_model=w, n_head=w // 64, d_ff=4 * w, vocab=case["vocab"])).to(torch.bfloat16)
            return model, torch.optim.AdamW(model.parameters(), lr=1e-4, weight_decay=0.01)
        model = ds2.DeepSpeech2(ds2.DS2Config(rnn_hidden=case["hidden"], rnn_layers=case["layers"]))
        model.rnn.flatten_parameters()
        return model, torch.optim.SGD(model.parameters(), lr=3e-4, momentum=0.9)


def prepare(case, seed):
    _join_group()
    torch.manual_seed(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    s = dict(case)
    if kind == "allreduce":
        s["x"] = _values(gen, case["numel"], _DTYPES[case["dtype"]])
    elif kind in ("emu_one_shot", "emu_two_shot"):
        n, ranks, dtype = case["numel"], case["ranks"], _DTYPES[case["dtype"]]
        nbytes = n * _SIZES[case["dtype"]]
        g = s["group"] = EmulatedGroup(ranks, nbytes)
        s["buffers"] = _buffers(g, dtype, n)
        for b in s["buffers"]:
            b.copy_(_values(gen, n, dtype))
        s["outs"] = [torch.empty(n, dtype=dtype, device="cuda") for _ in range(ranks)] if kind == "emu_one_shot" else None
        s["blocks"] = min(g.max_blocks(), max(1, -(-nbytes // (32 << 10))))
    elif kind == "emu_allgatherv":
        ranks, dtype = case["ranks"], _DTYPES[case["dtype"]]
        s["ins"] = [_values(gen, (r + 1) * case["rows"] * case["width"], dtype) for r in range(ranks)]
        total = sum(t.numel() for t in s["ins"])
        g = s["group"] = EmulatedGroup(ranks, total * _SIZES[case["dtype"]])
        s["buffers"] = _buffers(g, dtype, total)
        s["blocks"] = min(g.max_blocks(), 48)
    elif kind == "optimizer":
        model, base = _optimizer_model(case)
        s["model"] = model
        s["opt"], s["params"], s["flats"] = _wrap(model, base, gen)
        s["grads"] = [torch.empty_like(p).normal_(generator=gen).mul_(1e-2) for p in s["params"]]
    elif kind in ("gru_infer", "gru_train"):
        T, B, H = case["T"], case["B"], case["H"]
        with torch.device("cuda"):
            s["rnn"] = torch.nn.GRU(case["I"], H, num_layers=case["layers"], bidirectional=case["dirs"] == 2)
        s["x"] = torch.randn(T, B, case["I"], device="cuda", generator=gen)
        if kind == "gru_train":
            s["x"].requires_grad_(True)
            s["wrt"] = [s["x"]] + list(s["rnn"].parameters())
            s["dy"] = torch.randn(T, B, case["dirs"] * H, device="cuda", generator=gen) / (T * B)
    elif kind == "bn_clip":
        shape = (case["N"], case["C"], case["H"], case["W"])
        m = s["norm"] = BatchNormClip2d(case["C"], clip=_CLIP).cuda()
        with torch.no_grad():
            m.weight.uniform_(0.5, 1.5, generator=gen)
            m.bias.normal_(generator=gen)
        s["x"] = torch.randn(shape, device="cuda", generator=gen).mul_(2).add_(0.5).requires_grad_(True)
        s["dy"] = torch.randn(shape, device="cuda", generator=gen)
        s["wrt"] = [s["x"], m.weight, m.bias]
    else:
        cfg = ds2.DS2Config(n_frames=case["frames"], rnn_hidden=case["hidden"], rnn_layers=case["layers"], label_len=case["labels"])
        with torch.device("cuda"):
            model = ds2.DeepSpeech2(cfg)
        model.rnn.flatten_parameters()
        s["model"] = model
        s["opt"], _, s["flats"] = _wrap(model, torch.optim.SGD(model.parameters(), lr=3e-4, momentum=0.9), gen)
        s["batch_"] = (torch.randn(case["batch"], cfg.n_freq, cfg.n_frames, device="cuda", generator=gen),
                       torch.randint(1, cfg.n_classes, (case["batch"], cfg.label_len), device="cuda", generator=gen),
                       torch.full((case["batch"],), cfg.label_len, dtype=torch.long, device="cuda"))
    return s


def run(s):
    kind = s["kind"]
    if kind == "allreduce":
        return bc.allreduce(s["x"], average=s["average"])
    if kind in ("emu_one_shot", "emu_two_shot"):
        s["group"].allreduce(s["numel"], _DTYPES[s["dtype"]], kind[4:], outs=s["outs"], scale=1.0 / s["ranks"], blocks=s["blocks"])
        return s["outs"] or s["buffers"]
    if kind == "emu_allgatherv":
        s["group"].allgatherv(s["ins"], [0] * s["ranks"], blocks=s["blocks"])
        return s["buffers"]
    if kind == "optimizer":
        torch._foreach_copy_([p.grad for p in s["params"]], s["grads"])
        s["opt"].step()
        return s["flats"]
    if kind == "gru_infer":
        with torch.no_grad():
            return persistent_gru.gru_forward(s["rnn"], s["x"])
    if kind == "gru_train":
        y = persistent_gru.gru_forward(s["rnn"], s["x"])
        return [y.detach(), *torch.autograd.grad(y, s["wrt"], s["dy"])]
    if kind == "bn_clip":
        y = s["norm"](s["x"])
        grads = torch.autograd.grad(y, s["wrt"], s["dy"])
        return [y.detach(), s["norm"].running_mean, s["norm"].running_var, *grads]
    s["opt"].zero_grad()
    loss = s["model"].loss(*s["batch_"])
    loss.backward()
    s["opt"].step()
    return [loss.detach(), *s["flats"]]


def _parameters(case):
    """Number of parameters of the model of an `optimizer` or `ds2_step` case."""
    if case.get("model") == "resnet50":
        return 23508032 + 2049 * case["classes"]
    if case.get("model") == "gpt2":
        w = case["width"]
        return (case["vocab"] + 1024) * w + case["layers"] * (12 * w * w + 13 * w) + 2 * w
    h = case["hidden"]
    rnn = sum(2 * 3 * h * ((1312 if k == 0 else 2 * h) + h + 2) for k in range(case["layers"]))
    return 32 * 41 * 11 + 32 * 32 * 21 * 11 + 4 * 32 + rnn + 29 * (2 * h + 1)


def work(case):
    kind = case["kind"]
    es = _SIZES.get(case.get("dtype"), 4)
    if kind == "allreduce":
        return {"bytes": 2 * case["numel"] * es, "flops": case["numel"]}
    if kind in ("emu_one_shot", "emu_two_shot"):
        return {"bytes": 2 * case["ranks"] * case["numel"] * es, "flops": case["ranks"] * case["numel"]}
    if kind == "emu_allgatherv":
        total = case["ranks"] * (case["ranks"] + 1) // 2 * case["rows"] * case["width"] * es
        return {"bytes": total * (1 + case["ranks"]), "flops": 0}
    if kind == "optimizer":
        # gradient read, parameter read and written (16-bit ones written, their master copies read and written), state read and written
        per = {"resnet50": 2 + 2 + 8 + 8, "gpt2": 2 + 2 + 8 + 16, "ds2": 4 + 8 + 8}[case["model"]]
        n = _parameters(case)
        return {"bytes": per * n, "flops": 10 * n}
    if kind in ("gru_infer", "gru_train"):
        T, B, H, nd = case["T"], case["B"], case["H"], case["dirs"]
        weights = flops = 0
        for k in range(case["layers"]):
            width = (case["I"] if k == 0 else nd * H) + H
            weights += nd * 3 * H * (width + 2)
            flops += 2 * T * B * nd * 3 * H * width
        x, y = T * B * case["I"], T * B * nd * H
        if kind == "gru_infer":
            return {"bytes": 4 * (x + weights + y), "flops": flops}
        return {"bytes": 4 * (2 * x + 2 * weights + 2 * y), "flops": 3 * flops}
    if kind == "bn_clip":
        n = case["N"] * case["C"] * case["H"] * case["W"]
        return {"bytes": 4 * 4 * n, "flops": 20 * n}
    b, h = case["batch"], case["hidden"]
    t = (case["frames"] - 1) // 2 + 1
    n = _parameters(case)
    flops = 2 * b * 32 * t * (81 * 41 * 11 + 41 * 32 * 21 * 11)
    flops += sum(2 * t * b * 2 * 3 * h * ((1312 if k == 0 else 2 * h) + h) for k in range(case["layers"])) + 2 * t * b * 29 * 2 * h
    return {"bytes": 4 * (b * 161 * case["frames"] + 4 * n), "flops": 3 * flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("allreduce", "emu_allgatherv"):
        return "exact"                                   # values are copied
    if kind in ("emu_one_shot", "emu_two_shot"):
        return {"rel": 1e-6} if case["dtype"] == "fp32" else {"rel": 4e-3, "max": 2e-2}      # the order of the sums; one rounding to 16 bits
    if kind == "optimizer":
        return {"rel": 1e-5} if case["model"] == "ds2" else {"rel": 2e-3, "max": 2e-2}       # bf16 parameters: roundings that fall the other way
    if kind in ("gru_infer", "gru_train"):
        return {"rel": 3e-3}                             # TF32 operands (10-bit mantissas) through the recurrence
    if kind == "bn_clip":
        return {"rel": 2e-5, "max": 2e-3}                # fp32 sums over the batch; single elements at the edge of the clip
    return {"rel": 5e-3}                                 # TF32 through the whole model and back
