"""Fused layer of ranks on one GPU, calls that overlap.  The rows of a call release the kernel behind them when they start.  Where
that is the next call's GEMM, it sets up, and asks for its weights, under these rows, so weights that they are still writing
are the case to get right; where it is a collective, that the rows are its inputs.  No other kernel is released early: a GEMM
behind a collective starts at its end."""
import pytest
import torch

import yali_b200 as yali

pytestmark = pytest.mark.gpu

BF16 = torch.bfloat16


def rnd(shape, seed, std=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * std).to(BF16)


def layer(xs, ws, norm, res):
    h = sum(x.double() @ w.double().T for x, w in zip(xs, ws)) + res.double()
    return h, h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-5) * norm.double()


def close(got, want):
    # bf16 sums of the K splits, the row and the output: three roundings of at most 2^-9 each, and some room.
    assert ((got.double() - want).norm() / want.norm()).item() < 2.0 ** -7


@pytest.mark.parametrize("world", [2, 8])
@pytest.mark.parametrize("rows,width", [(256, 128), (384, 1024), (1024, 512)])
def test_weights_that_the_call_in_front_writes(world, rows, width):
    """The output of one call is the weight of the next: [rows, width] -> N = rows, K = width."""
    with yali.Comm.emulated(world, device=0) as c:
        norm, res, norm2 = rnd((width,), 1, 0.1) + 1, rnd((rows, width), 2), rnd((rows,), 3, 0.1) + 1
        w1 = [rnd((width, 128), 10 + r, 0.1) for r in range(world)]
        w2 = [torch.zeros((rows, width), dtype=BF16, device="cuda") for _ in range(world)]
        x2, res2 = [rnd((40, width), 30 + r, 0.1) for r in range(world)], rnd((40, rows), 4)
        out2 = [torch.empty((40, rows), dtype=BF16, device="cuda") for _ in range(world)]
        steps = [[rnd((rows, 128), 100 * s + r) for r in range(world)] for s in range(3)]
        torch.cuda.synchronize()
        got = []
        for x1 in steps:
            c.fused_linear_rmsnorm(x1, w1, [norm] * world, [res] * world, out=w2)
            c.fused_linear_rmsnorm(x2, w2, [norm2] * world, [res2] * world, out=out2)
            got.append((w2[0].clone(), [o.clone() for o in out2]))
        c.sync()
        for x1, (w, outs) in zip(steps, got):
            close(w, layer(x1, w1, norm, res)[1])
            want = layer(x2, [w] * world, norm2, res2)[1]  # every rank has the same weight
            for o in outs:
                close(o, want)


@pytest.mark.parametrize("world,rows,k,n", [(2, 8, 1024, 1024), (4, 33, 512, 640), (2, 300, 512, 1152), (8, 130, 256, 384)])
def test_weights_that_a_collective_in_front_writes(world, rows, k, n):
    with yali.Comm.emulated(world, device=0) as c:
        x, norm, res = [rnd((rows, k), 10 + r) for r in range(world)], rnd((n,), 1, 0.1) + 1, rnd((rows, n), 2)
        w = [torch.zeros((n, k), dtype=BF16, device="cuda") for _ in range(world)]
        parts = [[rnd((n, k), 50 * s + r, 0.05) for r in range(world)] for s in range(3)]
        pre = [torch.empty_like(res) for _ in range(world)]
        torch.cuda.synchronize()
        got = []
        for p in parts:
            c.all_reduce(p, w)
            y = c.fused_linear_rmsnorm(x, w, [norm] * world, [res] * world, residual_out=pre)
            got.append(([t.clone() for t in pre], y))
        c.sync()
        for p, (h, y) in zip(parts, got):
            total = sum(t.double() for t in p).to(BF16)
            want = layer(x, [total] * world, norm, res)
            for r in range(world):
                close(h[r], want[0])
                close(y[r], want[1])


def replayed(c, steps, graph, written):
    """Runs `steps` (calls without a kernel of another kind between them): in the stream, or captured and replayed twice, the tensors
    that it writes cleared in front of each."""
    if not graph:
        steps()
        return c.sync()
    steps()  # before the capture: what a call sets up once
    c.sync()
    g, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=side):
        steps()
    for _ in range(2):
        for t in written:
            t.zero_()
        g.replay()
    torch.cuda.synchronize()
    c.check()
    del g


@pytest.mark.parametrize("graph", [False, True])
# 3 x 128 and 100 x 384: rows of small CTAs, and a width whose last pair of columns is half empty; 50 x 3712: one tile of lines;
# 40 x 2048 with eight ranks: one tile, eight splits; 300 x 1152: several tiles.
@pytest.mark.parametrize("world,rows,k,n", [(2, 3, 256, 128), (4, 100, 320, 384), (2, 50, 1984, 3712), (8, 40, 1216, 2048), (2, 300, 512, 1152)])
def test_collectives_that_read_the_rows_in_front(world, rows, k, n, graph):
    """all_reduce, all_reduce_rmsnorm and reduce_scatter + all_gather of a layer's outputs, each directly behind a layer."""
    with yali.Comm.emulated(world, device=0, timeout_ms=2000) as c:
        w, norm, res = [rnd((n, k), 10 + r, 0.05) for r in range(world)], rnd((n,), 1, 0.1) + 1, rnd((rows, n), 2)
        shard = c.shard_elems(rows * n)

        def outs():
            return [torch.zeros((rows, n), dtype=BF16, device="cuda") for _ in range(world)]
        runs = [{"x": [rnd((rows, k), 50 * s + r) for r in range(world)], "out": outs(), "pre": outs(), "sum": outs(), "sum2": outs(),
                 "pre2": outs(), "shards": [torch.zeros(shard, dtype=BF16, device="cuda") for _ in range(world)]} for s in range(9)]
        torch.cuda.synchronize()

        def steps():
            for i, s in enumerate(runs):
                c.fused_linear_rmsnorm(s["x"], w, [norm] * world, [res] * world, out=s["out"], residual_out=s["pre"])
                if i % 3 == 0:
                    c.all_reduce(s["out"], s["sum"])
                elif i % 3 == 1:
                    c.all_reduce_rmsnorm(s["pre"], [norm] * world, s["out"], out=s["sum"], residual_out=s["pre2"])
                else:
                    c.reduce_scatter([t.view(-1) for t in s["out"]], s["shards"])
                    c.all_gather(s["shards"], rows * n, [t.view(-1) for t in s["sum"]])
        replayed(c, steps, graph, [t for s in runs for k, ts in s.items() if k != "x" for t in ts])
        for i, s in enumerate(runs):
            h, y = layer(s["x"], w, norm, res)
            for r in range(world):
                close(s["out"][r], y)
                close(s["pre"][r], h)
                # What was read is what the rows hold now: exact but for the rounding of the sum, or of the sum, the row and its norm.
                if i % 3 == 1:
                    want = sum(t.double() for t in s["pre"]) + s["out"][r].double()
                    close(s["pre2"][r], want)
                    close(s["sum"][r], want * torch.rsqrt(want.pow(2).mean(-1, keepdim=True) + 1e-5) * norm.double())
                else:
                    close(s["sum"][r], sum(t.double() for t in s["out"]))


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("world,many,width", [(2, 3000, 2176), (8, 1700, 1024)])
def test_calls_of_few_and_of_many_rows_take_turns(world, many, width, graph):
    """Rows above and below the size up to which they release the next call, in both orders; x, weights and residual of a call are
    the outputs of the one in front."""
    few = 24
    assert few * width * world < 12 << 20 < many * width * world
    with yali.Comm.emulated(world, device=0, timeout_ms=2000) as c:
        norm, w = rnd((width,), 1, 0.1) + 1, [rnd((width, 64), 10 + r, 0.1) for r in range(world)]
        norm2, w2 = rnd((width,), 2, 0.1) + 1, [rnd((width, width), 30 + r, 0.03) for r in range(world)]

        def outs(rows):
            return [torch.zeros((rows, width), dtype=BF16, device="cuda") for _ in range(world)]
        runs = [{"x": [rnd((many, 64), 50 * s + r) for r in range(world)], "x2": [rnd((few, width), 500 + 50 * s + r) for r in range(world)],
                 "res": rnd((many, width), 900 + s), "a": outs(many), "b": outs(few), "d": outs(few), "e": outs(many)} for s in range(3)]
        torch.cuda.synchronize()

        def steps():
            for s in runs:
                c.fused_linear_rmsnorm(s["x"], w, [norm] * world, [s["res"]] * world, out=s["a"])  # many
                # Few rows that are made of the many: x and residual, then the weights.
                c.fused_linear_rmsnorm([t[:few] for t in s["a"]], w2, [norm2] * world, [t[few:2 * few] for t in s["a"]], out=s["b"])
                c.fused_linear_rmsnorm(s["x2"], [t[:width] for t in s["a"]], [norm2] * world, s["b"], out=s["d"])
                c.fused_linear_rmsnorm(s["x"], w, [norm] * world, s["a"], out=s["e"])  # many again, behind few
        replayed(c, steps, graph, [t for s in runs for k in "abde" for t in s[k]])
        for s in runs:
            a = layer(s["x"], w, norm, s["res"])[1]
            for r in range(world):
                close(s["a"][r], a)
                close(s["b"][r], layer([t[:few] for t in s["a"]], w2, norm2, s["a"][r][few:2 * few])[1])
                close(s["d"][r], layer(s["x2"], [t[:width] for t in s["a"]], norm2, s["b"][r])[1])
                close(s["e"][r], layer(s["x"], w, norm, s["a"][r])[1])
