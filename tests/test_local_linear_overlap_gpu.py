"""Fused layer of ranks on one GPU, calls that overlap: a call's GEMM sets up, and asks for its weights, under the end of the
kernel in front of it, so weights that this kernel is still writing are the case to get right."""
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
