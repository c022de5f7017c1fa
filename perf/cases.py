"""The work a program on one GPU has this framework do, as measurable cases.

With one GPU the ranks of a group share it (`Comm.emulated`): one cooperative launch per call runs the CTAs
of all ranks.  Every case is one or two calls of the communicator on tensors the program already holds; sizes
are those of the benchmark, the tests and the Llama-style layer of this repository, or generic.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs on the GPU (pinned host memory for the host path) and the communicator
    run(state)           one pass; returns every rank's outputs
    work(case)           bytes and operations a pass cannot do without
    tolerance(case)      how far another correct implementation may be from the results
"""
import math

import torch

import yali_b200 as yali

DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
SIZE = {"fp32": 4, "fp16": 2, "bf16": 2}

# The widest traffic of a listed device case: two ranks, 128 MiB in and out each.
MOST_BYTES = 512 << 20


def listed():
    return [
        # The smallest message of the size sweeps: launches and latency are all there is.
        {"name": "ar-fp32-4KiB-w2", "kind": "all_reduce", "world": 2, "dtype": "fp32", "out": "fp32", "n": 1024, "scale": 1.0},
        # The latency headline of the benchmark.
        {"name": "ar-fp32-1MiB-w2", "kind": "all_reduce", "world": 2, "dtype": "fp32", "out": "fp32", "n": 262144, "scale": 1.0},
        # A medium message that is no multiple of any vector, slice or shard.
        {"name": "ar-fp16-ragged-w4", "kind": "all_reduce", "world": 4, "dtype": "fp16", "out": "fp16", "n": 3000017, "scale": 1.0},
        # The bandwidth headline of the benchmark.
        {"name": "ar-fp32-128MiB-w2", "kind": "all_reduce", "world": 2, "dtype": "fp32", "out": "fp32", "n": 33554432, "scale": 1.0},
        # Data-parallel training: a 25 MiB fp32 gradient bucket, averaged and handed on in bf16.
        {"name": "grad-fp32-bf16-25MiB-w8", "kind": "all_reduce", "world": 8, "dtype": "fp32", "out": "bf16", "n": 6553600, "scale": 0.125},
        # Sharded training: reduce-scatter of the gradients, all-gather of the shards, 64 MiB bf16.
        {"name": "rs-ag-bf16-64MiB-w4", "kind": "rs_ag", "world": 4, "dtype": "bf16", "n": 33554432},
        # Tensor-parallel decode of 16 tokens: all-reduce + residual + RMSNorm, hidden 4096.
        {"name": "norm-bf16-16x4096-w8", "kind": "norm", "world": 8, "dtype": "bf16", "rows": 16, "hidden": 4096},
        # The same step in prefill, 2048 tokens.
        {"name": "norm-bf16-2048x4096-w2", "kind": "norm", "world": 2, "dtype": "bf16", "rows": 2048, "hidden": 4096},
        # The fused row-parallel projection (o_proj of hidden 4096 over two ranks) in decode, 8 tokens.
        {"name": "linear-8x2048x4096-w2", "kind": "linear", "world": 2, "rows": 8, "k": 2048, "hidden": 4096},
        # down_proj over eight ranks (14336 / 8 = 1792) with a ragged batch of 300 tokens.
        {"name": "linear-300x1792x4096-w8", "kind": "linear", "world": 8, "rows": 300, "k": 1792, "hidden": 4096},
        # o_proj over two ranks in prefill, 2048 tokens.
        {"name": "linear-2048x2048x4096-w2", "kind": "linear", "world": 2, "rows": 2048, "k": 2048, "hidden": 4096},
        # Data that lives in pinned host memory, 32 MiB fp32 per rank: copy in, all-reduce, copy out.
        {"name": "host-fp32-32MiB-w2", "kind": "host", "world": 2, "dtype": "fp32", "n": 8388608},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["all_reduce", "all_reduce", "all_reduce", "rs_ag", "norm", "norm", "linear", "linear", "linear", "host"])
    world = rng.choice([2, 4, 8])
    if kind == "linear":
        # Rows up to 2048, slices of K up to a share of 14336 and at most 2048, widths that are multiples of 128.
        return {"kind": kind, "world": world, "rows": _log(rng, 1, 2048), "k": 64 * rng.randint(4, min(32, 224 // world)), "hidden": 128 * rng.randint(8, 32)}
    if kind == "norm":
        # Rows of whole 16-byte vectors.
        dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
        hidden = 128 * rng.randint(2, 64)
        most = min(4096, MOST_BYTES // (4 * world * hidden * SIZE[dtype]))
        return {"kind": kind, "world": world, "dtype": dtype, "rows": _log(rng, 1, most), "hidden": hidden}
    dtype = rng.choice(["fp32", "fp16", "bf16"])
    if kind == "host":
        return {"kind": kind, "world": 2, "dtype": dtype, "n": _log(rng, 65536, (32 << 20) // SIZE[dtype])}
    if kind == "rs_ag":
        return {"kind": kind, "world": world, "dtype": dtype, "n": _log(rng, 4096, MOST_BYTES // (2 * world * SIZE[dtype]))}
    # Half of the all-reduces also average and change the type, as gradient buckets do.
    out, scale = dtype, 1.0
    if rng.random() < 0.5:
        scale = 1.0 / world
        out = rng.choice({"fp32": ["fp32", "fp16", "bf16"], "fp16": ["fp16", "fp32"], "bf16": ["bf16", "fp32"]}[dtype])
    most = MOST_BYTES // (world * (SIZE[dtype] + SIZE[out]))
    return {"kind": kind, "world": world, "dtype": dtype, "out": out, "n": _log(rng, 256, most), "scale": scale}


_comms = {}


def _comm(world):
    """The program's one communicator of that size."""
    if world not in _comms:
        _comms[world] = yali.Comm.emulated(world, device=0)
    return _comms[world]


def _randn(gen, shape, dtype, std=1.0):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).mul_(std).to(dtype)


def prepare(case, seed):
    world, kind = case["world"], case["kind"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = {"kind": kind, "comm": _comm(world)}
    if kind == "linear":
        # Activations of unit size, weights of the usual 0.02, a residual stream that is alike on every rank.
        t, k, h = case["rows"], case["k"], case["hidden"]
        bf16 = torch.bfloat16
        s["x"] = [_randn(g, (t, k), bf16) for _ in range(world)]
        s["w"] = [_randn(g, (h, k), bf16, 0.02) for _ in range(world)]
        norm, res = _randn(g, (h,), bf16, 0.1) + 1, _randn(g, (t, h), bf16)
        s["norm"] = [norm.clone() for _ in range(world)]
        s["res"] = [res.clone() for _ in range(world)]
        s["res_out"] = [torch.empty_like(res) for _ in range(world)]
        return s
    dtype = DTYPES[case["dtype"]]
    if kind == "norm":
        shape = (case["rows"], case["hidden"])
        s["x"] = [_randn(g, shape, dtype) for _ in range(world)]
        norm, res = _randn(g, shape[1:], dtype, 0.1) + 1, _randn(g, shape, dtype)
        s["norm"] = [norm.clone() for _ in range(world)]
        s["res"] = [res.clone() for _ in range(world)]
        s["res_out"] = [torch.empty_like(res) for _ in range(world)]
        return s
    # Gradients and activations alike: normally distributed, of moderate size.
    xs = [_randn(g, (case["n"],), dtype) for _ in range(world)]
    if kind == "host":
        s["src"] = [torch.empty(x.shape, dtype=dtype, pin_memory=True).copy_(x) for x in xs]
        s["dst"] = [torch.empty(x.shape, dtype=dtype, pin_memory=True) for x in xs]
        return s
    s["x"] = xs
    if kind == "rs_ag":
        shard = s["comm"].shard_elems(case["n"])
        # The padding behind the message's end in the last shards is not written.
        s["shards"] = [torch.zeros(shard, dtype=dtype, device="cuda") for _ in range(world)]
        s["full"] = [torch.empty_like(x) for x in xs]
        s["n"] = case["n"]
        return s
    s["scale"] = case["scale"] if case["scale"] != 1.0 or case["out"] != case["dtype"] else None
    s["y"] = [torch.empty(case["n"], dtype=DTYPES[case["out"]], device="cuda") for _ in range(world)]
    return s


def run(s):
    comm, kind = s["comm"], s["kind"]
    if kind == "all_reduce":
        return comm.all_reduce(s["x"], s["y"], scale=s["scale"])
    if kind == "rs_ag":
        comm.reduce_scatter(s["x"], s["shards"])
        return {"shards": s["shards"], "full": comm.all_gather(s["shards"], s["n"], s["full"])}
    if kind == "norm":
        y = comm.all_reduce_rmsnorm(s["x"], s["norm"], s["res"], eps=1e-5, residual_out=s["res_out"])
        return {"y": y, "residual": s["res_out"]}
    if kind == "linear":
        y = comm.fused_linear_rmsnorm(s["x"], s["w"], s["norm"], s["res"], eps=1e-5, residual_out=s["res_out"])
        return {"y": y, "residual": s["res_out"]}
    return comm.all_reduce_host(s["src"], s["dst"])


def work(case):
    world, kind = case["world"], case["kind"]
    if kind == "linear":
        t, k, h = case["rows"], case["k"], case["hidden"]
        # x, W, residual, norm weight in; output and new residual out; bf16 throughout.
        return {"bytes": world * 2 * (t * k + h * k + t * h + h + 2 * t * h), "flops": world * 2 * t * k * h}
    if kind == "norm":
        n, b = case["rows"] * case["hidden"], SIZE[case["dtype"]]
        return {"bytes": world * b * (4 * n + case["hidden"]), "flops": world * n * (world + 5)}
    n, b = case["n"], SIZE[case["dtype"]]
    if kind == "rs_ag":
        # Every rank's message in, the shards out and in again, every rank's message out.
        return {"bytes": b * (2 * world * n + 2 * n), "flops": n * (world - 1)}
    out = SIZE[case["out"]] if kind == "all_reduce" else b
    return {"bytes": world * n * (b + out), "flops": n * (world - 1)}


def tolerance(case):
    kind = case["kind"]
    if kind == "linear":
        # The ranks' partial rows travel in bf16 (relative rounding 2^-9 each) before they are added.
        return {"rel": 1e-2}
    # One rounding of an fp32 sum to the output type, or the order of the additions in fp32.
    return {"rel": {"fp32": 1e-5, "fp16": 1e-3, "bf16": 5e-3}[case["out"] if kind == "all_reduce" else case["dtype"]]}
