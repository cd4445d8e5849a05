"""Performance cases of the codec: what a program that uses neuzip_b200 has it do.

Every case is one of seven kinds of call, over the sizes of the models this package is
used with (Llama-shaped blocks of 1.3B, 7B and 70B parameters and their tensor-parallel
shards) and over small, odd and ragged sizes:

    read       decompress stored matrices           Manager.read / Manager.read_many
    write      compress a matrix                    the C library's compress calls
    update     read, SGD step, write, read back     Manager.read / Manager.write
    linear     forward of a converted Linear        Manager.convert, module call
    fused      the same with the fused linear on    Manager.fuse_linear
    train      forward and backward of a Linear     Manager.convert, autograd
    embed      token lookup in a compressed table   Manager.convert, module call

Matrices are normal with a standard deviation of about 0.02 that differs a little from row
to row, which is what the projections of a trained transformer look like to the codec.
"""
import math

import torch

import neuzip_b200 as nz
from neuzip_b200 import _lib

# The seven projections of one block: 7B shape, and a 70B block split over eight GPUs.
_BLOCK_7B = ("4096x4096,4096x4096,4096x4096,4096x4096,11008x4096,11008x4096,4096x11008")
_SHARD_70B = ("1024x8192,128x8192,128x8192,8192x1024,3584x8192,3584x8192,8192x3584")


def listed():
    return [
        # one small matrix (a test model, an adapter): latency of a single call
        {"name": "read_small", "kind": "read", "shapes": "512x1024", "precision": 7, "normalizer": 0,
         "operand": True},
        # one attention projection of a 7B model, lossless: what every converted Linear does
        {"name": "read_matrix", "kind": "read", "shapes": "4096x4096", "precision": 7, "normalizer": 0,
         "operand": True},
        # a whole 7B block decoded ahead of its forward, lossless
        {"name": "read_block", "kind": "read", "shapes": _BLOCK_7B, "precision": 7, "normalizer": 0,
         "operand": True},
        # one rank's part of a 70B block at 3 mantissa bits (inference with lossy weights)
        {"name": "read_shard_s3", "kind": "read", "shapes": _SHARD_70B, "precision": 3, "normalizer": 0,
         "operand": True},
        # the most aggressive setting: no mantissa bits, block normaliser, a shape that fits nothing
        {"name": "read_ragged_s0", "kind": "read", "shapes": "4099x2051", "precision": 0,
         "normalizer": 512, "operand": False},
        # compressing one attention projection when a model is converted or a step is applied
        {"name": "write_matrix", "kind": "write", "shapes": "4096x4096", "precision": 7, "operand": True},
        # the largest matrix of a 70B model, lossy
        {"name": "write_large_s3", "kind": "write", "shapes": "8192x28672", "precision": 3,
         "operand": False},
        # the in-backward optimiser step of a 1.3B model: decompress, SGD, compress, next read
        {"name": "update_matrix", "kind": "update", "shapes": "2048x2048", "precision": 7},
        # one token through a converted Linear (batch-1 generation), default path
        {"name": "linear_token", "kind": "linear", "shapes": "4096x4096", "precision": 7, "rows": 1,
         "bias": False},
        # a small batch of generation with the fused decode -> tensor-core linear
        {"name": "linear_fused", "kind": "fused", "shapes": "11008x4096", "precision": 7, "rows": 16,
         "bias": False},
        # training: forward and backward of an up projection of a 1.3B model on 2048 tokens
        {"name": "train_linear", "kind": "train", "shapes": "5504x2048", "precision": 7, "rows": 2048,
         "bias": True},
        # a prompt of 512 tokens through a compressed embedding table
        {"name": "embed_prompt", "kind": "embed", "shapes": "32000x4096", "precision": 7, "rows": 512},
    ]


def _log_between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _operand_shape(rng, lo, hi):
    """A Linear weight: rows a multiple of 4, columns a multiple of 64."""
    return 4 * _log_between(rng, lo // 4, hi // 4), 64 * _log_between(rng, lo // 64, hi // 64)


def draw(rng):
    kind = rng.choice(("read", "read", "write", "update", "linear", "fused", "train", "embed"))
    precision = rng.choice((7, 7, 3, 1, 0))
    if kind in ("read", "write"):
        operand = rng.random() < 0.6
        count = 1 if kind == "write" else rng.choice((1, 1, 2, 4, 7))
        shapes, total = [], 0
        for _ in range(count):
            if operand:
                r, c = _operand_shape(rng, 256, 8192)
            else:
                r, c = _log_between(rng, 64, 8192), _log_between(rng, 64, 4096)
            total += r * c
            if not shapes or total <= 150_000_000:
                shapes.append(f"{r}x{c}")
        case = {"kind": kind, "shapes": ",".join(shapes), "precision": precision, "operand": operand}
        if kind == "read":
            case["normalizer"] = rng.choice((0, 0, 512)) if not operand and precision < 7 else 0
        return case
    if kind == "update":
        r, c = _operand_shape(rng, 512, 6144)
        return {"kind": kind, "shapes": f"{r}x{c}", "precision": precision}
    if kind == "embed":
        return {"kind": kind, "shapes": f"{_log_between(rng, 8000, 64000)}x{64 * rng.randint(8, 64)}",
                "precision": precision, "rows": _log_between(rng, 1, 1024)}
    # the fused linear needs a segment length that divides the columns: multiples of 1024 have one
    r, c = (_operand_shape(rng, 512, 5632) if kind != "fused"
            else (4 * _log_between(rng, 128, 3072), 1024 * rng.randint(1, 8)))
    rows = {"linear": (1, 512), "fused": (1, 256), "train": (256, 1536)}[kind]
    return {"kind": kind, "shapes": f"{r}x{c}", "precision": precision, "rows": _log_between(rng, *rows),
            "bias": rng.random() < 0.5}


# ------------------------------------------------------------------ inputs
def _shapes(case):
    return [tuple(int(d) for d in s.split("x")) for s in case["shapes"].split(",")]


def _weights(case, seed):
    """The case's matrices, bf16 on the GPU, from the seed alone."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = []
    for r, c in _shapes(case):
        scale = 0.02 * torch.exp(0.2 * torch.randn(r, 1, generator=g, device="cuda"))
        out.append(torch.randn(r, c, generator=g, device="cuda").mul_(scale).to(torch.bfloat16))
    return out, g


def _activations(case, seed):
    (w,), g = _weights(case, seed)
    r, c = w.shape
    x = torch.randn(case["rows"], c, generator=g, device="cuda").to(torch.bfloat16)
    bias = (torch.randn(r, generator=g, device="cuda") * 0.02).to(torch.bfloat16) if case["bias"] else None
    gy = torch.randn(case["rows"], r, generator=g, device="cuda").to(torch.bfloat16)
    return w, x, bias, gy


def _tokens(case, seed):
    (table,), g = _weights(case, seed)
    return table, torch.randint(0, table.shape[0], (1, case["rows"]), generator=g, device="cuda")


def _gradient(case, seed):
    (w,), g = _weights(case, seed)
    return w, (torch.randn(w.shape, generator=g, device="cuda") * 1e-3).to(torch.bfloat16)


def _converted(case, module):
    manager = nz.Manager(precision=case["precision"])
    if case["kind"] == "fused":
        manager.fuse_linear(256)
    model = manager.convert(torch.nn.Sequential(module))
    manager.total_size()          # as a program that reports the compressed size does
    return manager, model


def _dense_linear(w, bias):
    lin = torch.nn.Linear(w.shape[1], w.shape[0], bias=bias is not None, device="meta")
    lin.weight = torch.nn.Parameter(w)
    if bias is not None:
        lin.bias = torch.nn.Parameter(bias)
    return lin


def prepare(case, seed):
    kind = case["kind"]
    if kind == "read":
        manager = nz.Manager(precision=case["precision"], normalizer_size=case["normalizer"] or None)
        handles = [manager.write(w, operand=case["operand"]) for w in _weights(case, seed)[0]]
        manager.total_size()
        return {"kind": kind, "manager": manager, "handles": handles}
    if kind == "write":
        return _prepare_write(case, seed)
    if kind == "update":
        w, grad = _gradient(case, seed)
        manager = nz.Manager(precision=case["precision"])
        source = manager.write(w, operand=True)
        target = manager.write(w, operand=True)
        manager.total_size()
        return {"kind": kind, "manager": manager, "source": source, "target": target, "grad": grad}
    if kind == "embed":
        table, tokens = _tokens(case, seed)
        emb = torch.nn.Embedding(table.shape[0], table.shape[1], device="meta")
        emb.weight = torch.nn.Parameter(table)
        manager = nz.Manager(precision=case["precision"])
        module = nz.nn.Embedding(manager, emb)
        manager.total_size()
        return {"kind": kind, "module": module, "tokens": tokens}
    w, x, bias, gy = _activations(case, seed)
    manager, model = _converted(case, _dense_linear(w, bias))
    if kind == "train":
        x.requires_grad_(True)
    return {"kind": kind, "manager": manager, "module": model, "linear": model[0], "x": x, "gy": gy}


def _prepare_write(case, seed):
    lib = _lib.load()
    (w,), _ = _weights(case, seed)
    rows, cols = w.shape
    n, precision = w.numel(), case["precision"]
    lane = int(lib.nz_operand_lane_symbols_for(rows, cols, precision)) if case["operand"] else 0
    operand = lane != 0
    if operand:
        scratch_bytes = int(lib.nz_compress_operand_scratch_bytes(rows, cols, lane))
    else:
        lane = int(lib.nz_default_lane_symbols(precision))
        scratch_bytes = int(lib.nz_compress_scratch_bytes(n, lane))
    cap = int(lib.nz_container_bound(n, lane))
    return {
        "kind": "write", "lib": lib, "w": w, "operand": operand, "precision": precision, "lane": lane,
        "fractions": torch.zeros(int(lib.nz_frac_bytes(n, precision)), dtype=torch.uint8, device="cuda"),
        "container": torch.zeros(cap, dtype=torch.uint8, device="cuda"),
        "scratch": torch.empty(scratch_bytes, dtype=torch.uint8, device="cuda"),
    }


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "read":
        handles = state["handles"]
        if len(handles) == 1:
            return state["manager"].read(handles[0])
        return state["manager"].read_many(handles)
    if kind == "write":
        return _run_write(state)
    if kind == "update":
        manager = state["manager"]
        w = manager.read(state["source"])
        w.add_(state["grad"], alpha=-0.1)
        manager.write(w, state["target"])
        return {"weight": w, "stored": manager.read(state["target"])}
    if kind == "embed":
        return state["module"](state["tokens"])
    if kind in ("linear", "fused"):
        with torch.no_grad():
            return state["module"](state["x"])
    x, linear = state["x"], state["linear"]
    x.grad = None
    linear._p._gradient = None
    if linear.bias is not None:
        linear.bias.grad = None
    y = state["module"](x)
    y.backward(state["gy"])
    out = {"y": y.detach(), "dx": x.grad, "dw": linear._p._gradient}
    if linear.bias is not None:
        out["db"] = linear.bias.grad
    return out


def _run_write(s):
    lib, w = s["lib"], s["w"]
    stream = torch.cuda.current_stream().cuda_stream
    tail = (s["fractions"].data_ptr(), s["container"].data_ptr(), s["container"].numel(),
            s["scratch"].data_ptr(), s["scratch"].numel(), stream)
    if s["operand"]:
        _lib.check(lib.nz_compress_bf16_operand(w.data_ptr(), w.shape[0], w.shape[1], s["precision"],
                                                s["lane"], *tail))
    else:
        _lib.check(lib.nz_compress_bf16(w.data_ptr(), w.numel(), s["precision"], s["lane"], *tail))
    return {"container": s["container"], "fractions": s["fractions"]}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    s, kind = case["precision"], case["kind"]
    per_weight = (s + 1) / 8 + 2.6 / 8          # packed fractions + about 2.6 bits of coded exponent
    n = sum(r * c for r, c in _shapes(case))
    if kind in ("read", "write"):
        return {"bytes": n * (2 + per_weight), "flops": 0}
    if kind == "update":
        # stored weight and gradient in, updated weight and its stored form out, read back
        return {"bytes": n * (3 * per_weight + 3 * 2), "flops": 2 * n}
    if kind == "embed":
        return {"bytes": case["rows"] * _shapes(case)[0][1] * (2 + per_weight), "flops": 0}
    r, c = _shapes(case)[0]
    m = case["rows"]
    if kind in ("linear", "fused"):
        return {"bytes": n * per_weight + 2 * m * (r + c), "flops": 2 * m * n}
    return {"bytes": n * per_weight + 2 * n + 4 * m * (r + c), "flops": 6 * m * n}


def tolerance(case):
    if case["kind"] in ("read", "write", "update", "embed"):
        return "exact"
    # bf16 results of fp32 sums: one rounding each (0.0017 in the 2-norm), four times that;
    # a single element may be off by one unit in the last place of the largest results
    return {"rel": 7e-3, "max": 0.06}


# ------------------------------------------------------------------ the same in 64 bits
def _stored(w, precision):
    """What a lossy precision keeps of a bf16 tensor: the magnitude rounded half up at the cut."""
    if precision == 7:
        return w
    bits = w.view(torch.int16).to(torch.int32) & 0xFFFF
    drop = 7 - precision
    mag = (bits & 0x7FFF) + (1 << (drop - 1))
    mag = (mag >> drop) << drop
    out = (bits & 0x8000) | (mag & 0x7FFF)
    return torch.where(out >= 32768, out - 65536, out).to(torch.int16).view(torch.bfloat16)


def exact(case, seed):
    kind, precision = case["kind"], case["precision"]
    if kind == "read":
        if case["normalizer"]:
            return None
        out = [_stored(w, precision).double() for w in _weights(case, seed)[0]]
        return out[0] if len(out) == 1 else out
    if kind == "write":
        return None
    if kind == "update":
        w, grad = _gradient(case, seed)
        step = _stored(w, precision).double() - 0.1 * grad.double()
        return {"weight": step, "stored": step if precision == 7 else None}
    if kind == "embed":
        table, tokens = _tokens(case, seed)
        return _stored(table, precision)[tokens].double()
    w, x, bias, gy = _activations(case, seed)
    w64, x64, gy64 = _stored(w, precision).double(), x.double(), gy.double()
    y = x64 @ w64.t()
    if bias is not None:
        y = y + bias.double()
    if kind != "train":
        return y
    out = {"y": y, "dx": gy64 @ w64, "dw": gy64.t() @ x64}
    if bias is not None:
        out["db"] = gy64.sum(0)
    return out
