"""What the framework's users run, as measurable cases: embedding training steps and lookups, quantised
serving, the jagged copies, the input distribution's segment permutation, table quantisation and the
colour conversion, each through its public entry point, from a single request to a training batch.

A case is a dict of plain values; `kind` names the entry point, the rest are its sizes and options.
Inputs come from the seed alone and are made on the GPU.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from torchlib_xpu_b200 import cabi, load_torch_ops, tbe_modules

_DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
_TYPES = {"fp32": tbe_modules.SparseType.FP32, "fp16": tbe_modules.SparseType.FP16,
          "int8": tbe_modules.SparseType.INT8, "int4": tbe_modules.SparseType.INT4}
_ROW_ALIGN = 16


def listed():
    return [
        # One ranking request against quantised tables: a couple of candidates, every table looked up
        # a few times. What counts is the latency of a call.
        dict(name="serve_request", kind="serve", tables=26, rows=100_000, dims="64", types="int8", batch=2,
             len_lo=1, len_hi=20, alpha=1.05, pooling="sum", weighted=False, ids="int32", out="fp16"),
        # Offline scoring against 64 large quantised tables (the repository's quantised configuration: half
        # the tables INT8, half INT4).
        dict(name="serve_bulk", kind="serve", tables=64, rows=2_000_000, dims="128", types="int8,int4", batch=16384,
             len_lo=1, len_hi=100, alpha=1.1, pooling="sum", weighted=False, ids="int64", out="fp16"),
        # A forward pass without gradients over fp32 tables (the repository's first configuration).
        dict(name="lookup_fp32", kind="lookup", tables=8, rows=100_000, dims="128", weights="fp32", batch=2048,
             len_lo=1, len_hi=40, alpha=0.0, scattered=False, pooling="sum", weighted=False, ids="int64", out="fp32"),
        # A small training step, as in online training or a debugging run: few lookups, all launches.
        dict(name="train_small", kind="train", tables=8, rows=100_000, dims="64", weights="fp32", batch=256,
             len_lo=1, len_hi=10, alpha=1.05, scattered=True, pooling="sum", weighted=False, ids="int64", out="fp32",
             optimizer="adagrad"),
        # Tables of different widths, weighted mean pooling, plain SGD, 32-bit ids and a batch that is a
        # multiple of nothing.
        dict(name="train_mixed_widths", kind="train", tables=14, rows=250_007, dims="16,32,48,64,100,128,256",
             weights="fp32", batch=3001, len_lo=0, len_hi=30, alpha=1.05, scattered=True, pooling="mean",
             weighted=True, ids="int32", out="fp32", optimizer="sgd"),
        # The repository's training configuration: 26 fp16 tables, scattered Zipf ids, fp32 pooled rows
        # and gradients, row-wise Adagrad.
        dict(name="train_26_tables", kind="train", tables=26, rows=1_000_000, dims="128", weights="fp16", batch=8192,
             len_lo=1, len_hi=64, alpha=1.05, scattered=True, pooling="sum", weighted=False, ids="int64", out="fp32",
             optimizer="adagrad"),
        # A quarter of one GPU's share of the sharded configuration (the whole share does not fit three
        # times over): large tables, a large global batch, fp16 rows, pooled rows and gradients.
        dict(name="train_large_batch", kind="train", tables=16, rows=4_000_000, dims="128", weights="fp16", batch=65536,
             len_lo=1, len_hi=50, alpha=1.05, scattered=False, pooling="sum", weighted=False, ids="int64", out="fp16",
             optimizer="adagrad"),
        # Sequence features padded for attention, and the gradient back (the repository's jagged configuration).
        dict(name="jagged_pad", kind="jagged", op="pad", batch=4096, max_len=128, dim=256, dtype="fp32",
             offsets="int64"),
        # Position embeddings added to short odd-sized bf16 sequences.
        dict(name="jagged_add_odd", kind="jagged", op="add", batch=1023, max_len=77, dim=72, dtype="bf16",
             offsets="int64"),
        # A rank's ids and per-sample weights regrouped by owner before they are sent.
        dict(name="permute_ids", kind="permute", tables=128, batch=8192, len_lo=1, len_hi=50, ids="int64",
             lengths="int32", weighted=True, sum_given=True),
        # A trained table packed for serving and unpacked for a check.
        dict(name="quantise_table", kind="quantise", rows=2_000_000, dim=128, bits=8, dtype="fp32"),
        # One decoded 4K frame to RGB.
        dict(name="frame_4k", kind="frame", width=3840, height=2160, tiled=True, full_range=False),
    ]


# ---- drawn cases -------------------------------------------------------------------------------------
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, choices):
    return ",".join(str(d) for d in rng.sample(choices, rng.choice([1, 1, 1, 2, 3])))


def _fit(rng, lookups, tables, batch, len_hi):
    """A batch that keeps the expected lookups of all tables within `lookups`."""
    most = max(1, int(lookups / (tables * max(1.0, len_hi / 2))))
    return max(1, min(batch, most))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "lookup", "serve", "serve", "jagged", "jagged", "permute", "quantise",
                       "frame"])
    if kind in ("train", "lookup"):
        weights = rng.choice(["fp32", "fp16"])
        case = dict(kind=kind, tables=_log(rng, 1, 32), rows=_log(rng, 1000, 1_000_000),
                    dims=_dims(rng, [16, 32, 64, 96, 128, 128, 128, 200, 256]), weights=weights, len_lo=rng.choice([0, 1]),
                    len_hi=_log(rng, 2, 64), alpha=rng.choice([0.0, 1.05, 1.05]), scattered=rng.random() < 0.5,
                    pooling=rng.choice(["sum", "sum", "mean"]), weighted=rng.random() < 0.25,
                    ids=rng.choice(["int64", "int32"]), out="fp32" if weights == "fp32" else rng.choice(["fp32", "fp16"]))
        case["batch"] = _fit(rng, 8_000_000, case["tables"], _log(rng, 16, 32768), case["len_hi"])
        if kind == "train":
            case["optimizer"] = rng.choice(["adagrad", "adagrad", "sgd"])
        return case
    if kind == "serve":
        case = dict(kind="serve", tables=_log(rng, 1, 64), rows=_log(rng, 1000, 1_000_000),
                    dims=_dims(rng, [32, 64, 64, 128, 128, 256]), types=rng.choice(["int8", "int4", "int8,int4"]),
                    len_lo=rng.choice([0, 1]), len_hi=_log(rng, 2, 100), alpha=rng.choice([0.0, 1.05, 1.1]),
                    pooling=rng.choice(["sum", "sum", "mean"]), weighted=rng.random() < 0.25,
                    ids=rng.choice(["int64", "int32"]), out=rng.choice(["fp16", "fp16", "fp32"]))
        case["batch"] = _fit(rng, 16_000_000, case["tables"], _log(rng, 1, 16384), case["len_hi"])
        return case
    if kind == "jagged":
        dim = rng.choice([8, 33, 64, 72, 128, 200, 256, 512])
        max_len = _log(rng, 4, 512)
        return dict(kind="jagged", op=rng.choice(["pad", "unpad", "add"]), max_len=max_len, dim=dim,
                    batch=max(1, min(_log(rng, 8, 4096), (1 << 27) // (dim * max_len))),
                    dtype=rng.choice(["fp32", "fp16", "bf16"]), offsets=rng.choice(["int64", "int32"]))
    if kind == "permute":
        tables, len_hi = _log(rng, 2, 256), _log(rng, 2, 100)
        return dict(kind="permute", tables=tables, batch=_fit(rng, 26_000_000, tables, _log(rng, 8, 16384), len_hi),
                    len_lo=rng.choice([0, 1]), len_hi=len_hi, ids=rng.choice(["int64", "int32"]),
                    lengths=rng.choice(["int32", "int64"]), weighted=rng.random() < 0.5, sum_given=rng.random() < 0.7)
    if kind == "quantise":
        return dict(kind="quantise", rows=_log(rng, 1000, 2_000_000), dim=rng.choice([32, 64, 96, 128, 256]),
                    bits=rng.choice([8, 4]), dtype=rng.choice(["fp32", "fp16"]))
    width, height = rng.choice([(640, 360), (854, 480), (1280, 720), (1920, 1080), (2560, 1440), (3840, 2160)])
    return dict(kind="frame", width=width, height=height, tiled=rng.random() < 0.5, full_range=rng.random() < 0.3)


# The modules' small index tables outlive them, as in a program that keeps its modules: no set of tables
# is ever found at the address of an earlier one.
_index_tables = []


# ---- inputs ------------------------------------------------------------------------------------------
def _table_dims(case):
    """Widths of the tables: the case's list, over and over."""
    dims = [int(d) for d in case["dims"].split(",")]
    return [dims[t % len(dims)] for t in range(case["tables"])]


def _bag_lengths(gen, count, lo, hi):
    """Lengths spread evenly over lo..hi, in random order: a case's total does not depend on the seed."""
    spread = lo + torch.arange(count, device="cuda", dtype=torch.int64) * (hi - lo + 1) // count
    return spread[torch.randperm(count, device="cuda", generator=gen)]


def _offsets(lengths, dtype):
    off = torch.zeros(lengths.numel() + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lengths, 0, out=off[1:])
    return off.to(dtype)


def _row_ids(gen, rows, alpha, count, scattered=False):
    """Uniform row ids (alpha 0), or bounded Zipf ones by the inverse of the integral of x^-alpha, as
    hashed ids (`scattered`: the frequent rows lie anywhere in the table) or as ids sorted by frequency."""
    if alpha == 0:
        return torch.randint(0, rows, (count,), device="cuda", generator=gen)
    lo, hi = 0.5 ** (1 - alpha), (rows + 0.5) ** (1 - alpha)
    ids = torch.empty(count, dtype=torch.int64, device="cuda")
    step = 1 << 24
    for a in range(0, count, step):
        b = min(count, a + step)
        u = torch.rand(b - a, device="cuda", dtype=torch.float64, generator=gen)
        ids[a:b] = ((u * (hi - lo) + lo) ** (1 / (1 - alpha)) - 0.5).long().clamp_(0, rows - 1)
    if scattered:
        ids = torch.randperm(rows, device="cuda", generator=gen)[ids]
    return ids


def _lookup_inputs(case, gen):
    idt = torch.int64 if case["ids"] == "int64" else torch.int32
    lengths = _bag_lengths(gen, case["tables"] * case["batch"], case["len_lo"], case["len_hi"])
    offsets = _offsets(lengths, idt)
    count = int(offsets[-1].item())
    ids = _row_ids(gen, case["rows"], case["alpha"], count, case.get("scattered", False)).to(idt)
    weights = torch.rand(count, device="cuda", generator=gen) + 0.5 if case["weighted"] else None
    return dict(indices=ids, offsets=offsets, weights=weights)


def _prepare_tables(case, gen):
    dims, rows = _table_dims(case), case["rows"]
    dtype = _DTYPES[case["weights"]]
    w = torch.empty(rows * sum(dims), dtype=dtype, device="cuda").uniform_(-0.01, 0.01, generator=gen)
    adagrad = case.get("optimizer") == "adagrad"
    # a state in mid-training: squared gradients have been summed for a while
    m = torch.rand(rows * len(dims), device="cuda", generator=gen) * 1e-3 + 1e-5 if adagrad else None
    kinds = tbe_modules.OptimType
    module = tbe_modules.SplitTableBatchedEmbeddingBagsCodegen(
        [(rows, d) for d in dims], optimizer=kinds.EXACT_ROWWISE_ADAGRAD if adagrad else kinds.EXACT_SGD,
        learning_rate=0.01, eps=1e-8, pooling_mode=tbe_modules.PoolingMode[case["pooling"].upper()],
        weights_precision=_TYPES[case["weights"]], output_dtype=_TYPES[case["out"]], weights_dev=w, momentum1_dev=m)
    _index_tables.append(module.hash_size_cumsum)
    state = dict(module=module, **_lookup_inputs(case, gen))
    if case["kind"] == "train":
        grad = torch.randn((case["batch"], sum(dims)), device="cuda", generator=gen) * 0.01
        state["grad"] = grad.to(_DTYPES[case["out"]])
    return state


def _prepare_serve(case, gen):
    dims, rows = _table_dims(case), case["rows"]
    names = case["types"].split(",")
    specs = [(rows, d, _TYPES[names[t % len(names)]]) for t, d in enumerate(dims)]
    module = tbe_modules.IntNBitTableBatchedEmbeddingBagsCodegen(
        specs, pooling_mode=tbe_modules.PoolingMode[case["pooling"].upper()], output_dtype=_TYPES[case["out"]],
        row_alignment=_ROW_ALIGN)
    # tables of quantised rows as they lie in memory: any codes behind an fp16 {scale, bias} of a row
    # of values in [-0.1, 0.1]
    words = module.weights_dev.view(torch.int32) if module.weights_dev.numel() % 4 == 0 else None
    if words is None:
        raise ValueError("tables are whole 4-byte words")
    step = 1 << 29
    for a in range(0, words.numel(), step):
        words[a:a + step].random_(-(1 << 31), (1 << 31) - 1, generator=gen)
    for t, (r, d, ty) in enumerate(specs):
        stride = module.row_strides[t]
        start = module._w_off_host[t]
        table = module.weights_dev[start:start + r * stride].view(r, stride)
        levels = 255 if ty == tbe_modules.SparseType.INT8 else 15
        lo = -0.1 * (torch.rand(r, device="cuda", generator=gen) * 0.5 + 0.5)
        header = torch.stack([(0.1 - lo) / levels, lo], 1).half().contiguous().view(torch.uint8)
        table[:, :4] = header.view(r, 4)
    _index_tables.append(module.weights_offsets)
    return dict(module=module, **_lookup_inputs(case, gen))


def _prepare_jagged(case, gen):
    lengths = _bag_lengths(gen, case["batch"], 0, case["max_len"])
    off = _offsets(lengths, torch.int64 if case["offsets"] == "int64" else torch.int32)
    total, dtype = int(off[-1].item()), _DTYPES[case["dtype"]]
    make = lambda *shape: torch.randn(shape, device="cuda", generator=gen).to(dtype)  # noqa: E731
    padded = (case["batch"], case["max_len"], case["dim"])
    state = dict(offsets=off, total=total, max_len=case["max_len"], op=case["op"])
    if case["op"] != "unpad":
        state["values"] = make(total, case["dim"]).requires_grad_()
    if case["op"] != "pad":
        state["dense"] = make(*padded).requires_grad_()
    state["grad"] = make(total, case["dim"]) if case["op"] == "unpad" else make(*padded)
    return state


def _prepare_permute(case, gen):
    tables, batch = case["tables"], case["batch"]
    lengths = _bag_lengths(gen, tables * batch, case["len_lo"], case["len_hi"])
    total = int(lengths.sum().item())
    idt = torch.int64 if case["ids"] == "int64" else torch.int32
    ids = torch.randint(0, 1_000_000, (total,), device="cuda", generator=gen).to(idt)
    weights = torch.rand(total, device="cuda", generator=gen) if case["weighted"] else None
    order = torch.randperm(tables, device="cuda", generator=gen).to(torch.int32)
    lengths = lengths.view(tables, batch).to(torch.int32 if case["lengths"] == "int32" else torch.int64)
    return dict(order=order, lengths=lengths, ids=ids, weights=weights, total=total if case["sum_given"] else None)


def _prepare_frame(case, gen):
    # a decoder's surface: rows padded to the tiles' 128 bytes, planes to 32 rows
    stride = -(-case["width"] // 128) * 128
    rows_y, rows_uv = -(-case["height"] // 32) * 32, -(-(case["height"] // 2) // 32) * 32
    plane = lambda rows: torch.randint(0, 256, (rows * stride,), device="cuda", generator=gen, dtype=torch.uint8)  # noqa: E731
    return dict(y=plane(rows_y), uv=plane(rows_uv), stride=stride, case=case)


def prepare(case, seed):
    load_torch_ops()
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind = case["kind"]
    if kind in ("train", "lookup"):
        state = _prepare_tables(case, gen)
    elif kind == "serve":
        state = _prepare_serve(case, gen)
    elif kind == "jagged":
        state = _prepare_jagged(case, gen)
    elif kind == "permute":
        state = _prepare_permute(case, gen)
    elif kind == "quantise":
        x = torch.randn((case["rows"], case["dim"]), device="cuda", generator=gen) * 0.05
        state = dict(x=x.to(_DTYPES[case["dtype"]]), bits=case["bits"], half=case["dtype"] == "fp16")
    elif kind == "frame":
        state = _prepare_frame(case, gen)
    else:
        raise ValueError("unknown kind %r" % (kind,))
    state["kind"] = kind
    return state


# ---- one pass ----------------------------------------------------------------------------------------
def _run_train(s):
    module = s["module"]
    out = module(s["indices"], s["offsets"], s["weights"])
    out.backward(s["grad"])
    updated = [module.weights_dev.detach()]
    return [out.detach(), *updated, *([module.momentum1_dev] if module.momentum1_dev.numel() else [])]


@torch.no_grad()
def _run_lookup(s):
    return s["module"](s["indices"], s["offsets"], s["weights"])


def _run_jagged(s):
    ops = torch.ops.fbgemm
    leaves = [t for t in (s.get("values"), s.get("dense")) if t is not None]
    if s["op"] == "pad":
        out = ops.jagged_to_padded_dense(s["values"], [s["offsets"]], [s["max_len"]], 0.0)
    elif s["op"] == "unpad":
        out, _ = ops.dense_to_jagged(s["dense"], [s["offsets"]], s["total"])
    else:
        out = ops.jagged_dense_elementwise_add(s["values"], [s["offsets"]], s["dense"])
    return [out.detach(), *torch.autograd.grad(out, leaves, s["grad"])]


def _run_permute(s):
    return list(torch.ops.fbgemm.permute_2D_sparse_data(s["order"], s["lengths"], s["ids"], s["weights"], s["total"]))


def _run_quantise(s):
    packed = torch.ops.fbgemm.FloatOrHalfToFusedNBitRowwiseQuantizedSBHalf(s["x"], s["bits"])
    back = torch.ops.fbgemm.FusedNBitRowwiseQuantizedSBHalfToFloatOrHalf(packed, s["bits"], 1 if s["half"] else 0)
    return [packed, back]


def _run_frame(s):
    c = s["case"]
    return cabi.nv12_to_rgb(s["y"], s["uv"], c["width"], c["height"], s["stride"], c["full_range"], c["tiled"])


_RUN = dict(train=_run_train, lookup=_run_lookup, serve=_run_lookup, jagged=_run_jagged, permute=_run_permute,
            quantise=_run_quantise, frame=_run_frame)


def run(state):
    return _RUN[state["kind"]](state)


# ---- what a pass cannot do without -------------------------------------------------------------------
def _distinct(rows, alpha, count):
    """Expected distinct ids among `count` draws."""
    if alpha == 0:
        return rows * -math.expm1(count * math.log1p(-1.0 / rows))
    p = np.arange(1, rows + 1, dtype=np.float64) ** (-alpha)
    p /= p.sum()
    return float(-np.expm1(count * np.log1p(-p)).sum())


def work(case):
    """Expected bytes: every input read once, every output written once (a training step reads and
    writes the rows it touches, and their optimizer state)."""
    kind = case["kind"]
    if kind in ("train", "lookup", "serve"):
        dims, bags = _table_dims(case), case["tables"] * case["batch"]
        per_table = case["batch"] * (case["len_lo"] + case["len_hi"]) / 2
        lookups = per_table * case["tables"]
        distinct = _distinct(case["rows"], case["alpha"], per_table)
        idb = 8 if case["ids"] == "int64" else 4
        outb = _DTYPES[case["out"]].itemsize
        pooled = case["batch"] * sum(dims) * outb
        common = lookups * (idb + (4 if case["weighted"] else 0)) + (bags + 1) * idb + pooled
        flops = 2.0 * per_table * sum(dims)
        if kind == "serve":
            names = case["types"].split(",")
            row = sum(4 + d * (8 if names[t % len(names)] == "int8" else 4) // 8 for t, d in enumerate(dims))
            return {"bytes": common + distinct * row, "flops": flops}
        row = sum(dims) * _DTYPES[case["weights"]].itemsize
        if kind == "lookup":
            return {"bytes": common + distinct * row, "flops": flops}
        state = 8 * case["tables"] if case["optimizer"] == "adagrad" else 0
        return {"bytes": common + pooled + distinct * (2 * row + state), "flops": 2 * flops}
    if kind == "jagged":
        item = _DTYPES[case["dtype"]].itemsize
        padded = case["batch"] * case["max_len"] * case["dim"] * item
        # the backward passes read and write the positions inside the lengths
        jag = padded / 2
        bytes_ = {"pad": jag + padded + 2 * jag, "unpad": 2 * jag + jag + padded, "add": jag + 2 * padded + 2 * jag}[case["op"]]
        return {"bytes": bytes_, "flops": padded / item if case["op"] == "add" else 0}
    if kind == "permute":
        lookups = case["tables"] * case["batch"] * (case["len_lo"] + case["len_hi"]) / 2
        elem = (8 if case["ids"] == "int64" else 4) + (4 if case["weighted"] else 0)
        lens = case["tables"] * case["batch"] * (4 if case["lengths"] == "int32" else 8)
        return {"bytes": 2 * lookups * elem + 2 * lens, "flops": 0}
    if kind == "quantise":
        item = _DTYPES[case["dtype"]].itemsize
        packed = case["dim"] * case["bits"] // 8 + 4
        return {"bytes": case["rows"] * (2 * case["dim"] * item + 2 * packed), "flops": 0}
    return {"bytes": case["width"] * case["height"] * 4.5, "flops": 0}


def tolerance(case):
    """Sums of fp32 terms in another order; results that are stored as fp16 may round the other way.
    Copies, permutations, codes and colours are the same bytes."""
    if case["kind"] not in ("train", "lookup", "serve"):
        return "exact"
    half = case["out"] == "fp16" or case.get("weights") == "fp16"
    return {"rel": 1e-3, "max": 4e-3} if half else {"rel": 2e-6, "max": 5e-5}
