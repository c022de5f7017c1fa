"""Automatically chosen calls of a group whose ranks share one GPU run in one launch that exchanges nothing
(csrc/kernels/local_group.cu).  Inputs are small whole numbers, so every sum is exact in every type and results
are compared bit by bit; sizes sit at the edges of the 16-byte units, CTAs (512 units) and shards."""
import json
import mmap
import os
import subprocess
import sys

import pytest
import torch

import yali_b200 as yali

pytestmark = pytest.mark.gpu

ONE_LAUNCH = 1 << 9
WIDE_STORES = 1 << 11
F32, F16, BF16 = torch.float32, torch.float16, torch.bfloat16


@pytest.fixture(scope="module", params=[1, 2, 3, 4, 8])
def comm(request):
    c = yali.Comm.emulated(request.param, device=0)
    yield c
    c.close()


def whole(shape, dtype, seed, off=0):
    """Whole numbers in [-8, 8] in a buffer that starts `off` elements behind a 16-byte boundary."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randint(-8, 9, shape, generator=g, device="cuda").to(dtype)
    buf = torch.empty(x.numel() + off, dtype=dtype, device="cuda")[off:].view(x.shape)
    return buf.copy_(x)


def total(xs):
    return torch.stack([x.double() for x in xs]).sum(0)


@pytest.mark.parametrize("src,dst", [(F32, F32), (F16, F16), (BF16, BF16), (F32, BF16), (F32, F16), (BF16, F32), (F16, F32)])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 2047, 2048, 2049, 4095, 4097, 100003])
def test_sum(comm, src, dst, n):
    for off in (0, 1):
        xs = [whole((n,), src, 10 * n + r, off if r == comm.world - 1 else 0) for r in range(comm.world)]
        ys = comm.all_reduce(xs, scale=0.5, out_dtype=dst)
        assert comm.last_call()["flags"] & ONE_LAUNCH
        for y in ys:
            assert torch.equal(y.double(), total(xs) * 0.5)
    if src == dst:  # in place
        want = total(xs)
        comm.all_reduce(xs, xs)
        assert comm.last_call()["flags"] & ONE_LAUNCH and all(torch.equal(x.double(), want) for x in xs)


@pytest.mark.parametrize("src,dst", [(BF16, F32), (F16, F32), (F32, BF16), (F32, F16)])
@pytest.mark.parametrize("n", [8, 15, 4096, 4103, 400003, 3000001])
def test_sum_to_another_width_on_and_off_32_byte_boundaries(comm, src, dst, n):
    """Units of 32 bytes are stored in one access where every buffer allows it; one rank's input or output starts 16 bytes behind such a boundary."""
    size = lambda t: torch.empty(0, dtype=t).element_size()  # noqa: E731
    for in_off, out_off in ((0, 0), (16 // size(src), 0), (0, 16 // size(dst))):
        xs = [whole((n,), src, n + r, in_off if r == 0 else 0) for r in range(comm.world)]
        ys = [whole((n + 8,), dst, 1, out_off if r == comm.world - 1 else 0) for r in range(comm.world)]
        tails = [y[n:].clone() for y in ys]
        comm.all_reduce(xs, [y[:n] for y in ys], scale=0.5)
        assert comm.last_call()["flags"] & ONE_LAUNCH
        want = total(xs) * 0.5
        for y, tail in zip(ys, tails):
            assert torch.equal(y[:n].double(), want) and torch.equal(y[n:], tail)


@pytest.mark.parametrize("src,dst", [(BF16, F32), (F16, F32), (F32, BF16)])
def test_32_byte_stores_ask_for_outputs_on_32_byte_boundaries_only(comm, src, dst):
    n, size = 4103, lambda t: torch.empty(0, dtype=t).element_size()  # noqa: E731
    for in_off, out_off in ((0, 0), (16 // size(src), 0), (0, 16 // size(dst))):
        xs = [whole((n,), src, n + r, in_off if r == 0 else 0) for r in range(comm.world)]
        ys = [whole((n,), dst, 1, out_off if r == comm.world - 1 else 0) for r in range(comm.world)]
        comm.all_reduce(xs, ys)
        flags = comm.last_call()["flags"]
        assert flags & ONE_LAUNCH and bool(flags & WIDE_STORES) == (dst == F32 and out_off == 0)
        assert all(torch.equal(y.double(), total(xs)) for y in ys)


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("n", [1, 16, 17, 129, 8192, 65535, 65537])
def test_halves(comm, dtype, n):
    W, S = comm.world, comm.shard_elems(n) if comm.world > 1 else n
    xs = [whole((n,), dtype, n + r) for r in range(W)]
    want = total(xs)
    shards = comm.reduce_scatter(xs)
    assert comm.last_call()["flags"] & ONE_LAUNCH
    for r, s in enumerate(shards):
        part = want[min(n, r * S):min(n, (r + 1) * S)]
        assert torch.equal(s[:part.numel()].double(), part)
    for f in comm.all_gather(shards, n):
        assert torch.equal(f.double(), want)
    assert comm.last_call()["flags"] & ONE_LAUNCH
    # Every rank's shard at its place inside the rank's own message: both halves in place.
    if n % (16 * W) == 0:
        views = [x[r * S:(r + 1) * S] for r, x in enumerate(xs)]
        comm.reduce_scatter(xs, views)
        comm.all_gather(views, n, xs)
        assert comm.last_call()["flags"] & ONE_LAUNCH and all(torch.equal(x.double(), want) for x in xs)


@pytest.mark.parametrize("dtype", [F32, F16, BF16])
@pytest.mark.parametrize("rows,hidden", [(1, 8), (3, 4096), (16, 4104), (200, 1000), (300, 4096), (40, 8192), (160, 8192)])
def test_norm(comm, dtype, rows, hidden):
    W = comm.world
    xs = [whole((rows, hidden), dtype, r) for r in range(W)]
    res = [whole((rows, hidden), dtype, 50 + r) for r in range(W)]  # not alike on the ranks: each uses its own
    ws = [whole((hidden,), dtype, 90 + r) for r in range(W)]
    pre = [torch.empty_like(x) for x in xs]
    ys = comm.all_reduce_rmsnorm(xs, ws, res, eps=1e-5, residual_out=pre)
    assert comm.last_call()["flags"] & ONE_LAUNCH
    plain = comm.all_reduce_rmsnorm(xs, ws, None, eps=1e-5)
    # The rows are exact; what is left is the fp32 sum of squares and product (a few 2^-23) and one rounding.
    rtol = {F32: 2e-6, F16: 2.0 ** -10, BF16: 2.0 ** -7}[dtype]
    for r in range(W):
        s = total(xs) + res[r].double()
        assert torch.equal(pre[r].double(), s)
        for got, row in ((ys[r], s), (plain[r], total(xs))):
            ref = row * torch.rsqrt(row.pow(2).mean(-1, keepdim=True) + 1e-5) * ws[r].double()
            torch.testing.assert_close(got.double(), ref, rtol=rtol, atol=1e-6)
    # The multi-GPU kernel on request, and for outputs that lie on the inputs of several ranks.
    again = comm.all_reduce_rmsnorm(xs, ws, res, eps=1e-5, mode="flash")
    assert not comm.last_call()["flags"] & ONE_LAUNCH
    torch.testing.assert_close(again[0].double(), ys[0].double(), rtol=2 * rtol, atol=1e-6)
    if rows * hidden < 65536:
        comm.all_reduce_rmsnorm(xs, ws, res, eps=1e-5, out=xs)
        assert not comm.last_call()["flags"] & ONE_LAUNCH
        torch.testing.assert_close(xs[0].double(), ys[0].double(), rtol=2 * rtol, atol=1e-6)


# The cuts of the norm kernel: one, two or four ranks per CTA, weights ahead of the barrier and behind it, one to four vectors per thread, rows
# that do not fill their last warp.  Groups of 2, 4 and 8 change the cut at different rows, so every group runs all of them.
@pytest.mark.parametrize("dtype,hidden,rows", [(BF16, 2944, (40, 90, 300, 900)), (F16, 24, (5, 2000, 20000)), (BF16, 8192, (3, 30, 400)),
                                               (F32, 4096, (20, 130, 400)), (F32, 8192, (9, 250)), (BF16, 12296, (9, 300)), (F32, 1000, (37, 1300))])
def test_cuts_of_the_norm(comm, dtype, hidden, rows):
    W, rtol = comm.world, {F32: 2e-6, F16: 2.0 ** -10, BF16: 2.0 ** -7}[dtype]
    ws = [whole((hidden,), dtype, 90 + r) for r in range(W)]
    for n in rows:
        xs, res = [whole((n, hidden), dtype, r) for r in range(W)], [whole((n, hidden), dtype, 50 + r) for r in range(W)]
        pre = [torch.empty_like(x) for x in xs]
        ys = comm.all_reduce_rmsnorm(xs, ws, res, eps=1e-5, residual_out=pre)
        assert comm.last_call()["kernel"] == "local_norm"
        s = total(xs)
        for r in range(W):
            row = s + res[r].double()
            assert torch.equal(pre[r].double(), row)
            ref = row * torch.rsqrt(row.pow(2).mean(-1, keepdim=True) + 1e-5) * ws[r].double()
            torch.testing.assert_close(ys[r].double(), ref, rtol=rtol, atol=1e-6)
        # In place: the residual stream is its own output.
        keep = [t.clone() for t in res]
        comm.all_reduce_rmsnorm(xs, ws, keep, eps=1e-5, residual_out=keep)
        assert all(torch.equal(k, p) for k, p in zip(keep, pre))


@pytest.mark.parametrize("world", [5, 6, 7])
@pytest.mark.parametrize("dtype,hidden,rows", [(BF16, 2944, (40, 200, 800)), (F16, 8192, (10, 300)), (F32, 8192, (9, 150)), (F32, 1000, (37, 1300))])
def test_norm_of_odd_groups(world, dtype, hidden, rows):
    with yali.Comm.emulated(world, device=0) as c:
        test_cuts_of_the_norm(c, dtype, hidden, rows)


@pytest.mark.parametrize("dtype", [F32, F16, BF16])
@pytest.mark.parametrize("rows,hidden", [(1, 4096), (16, 4096), (5, 1024), (3, 8192), (128, 4096), (7, 256)])
def test_norm_of_the_one_shot_kernel(comm, dtype, rows, hidden):
    """The row epilogue of the multi-GPU kernel, three calls back to back: each rank with a residual and a weight of its own."""
    if comm.world == 1:
        pytest.skip("a group of one has nothing to send")
    W, rtol = comm.world, {F32: 2e-6, F16: 2.0 ** -10, BF16: 2.0 ** -7}[dtype]
    xs, res = [whole((rows, hidden), dtype, r) for r in range(W)], [whole((rows, hidden), dtype, 50 + r) for r in range(W)]
    ws = [whole((hidden,), dtype, 90 + r) for r in range(W)]
    pre = [[torch.empty_like(x) for x in xs] for _ in range(3)]
    ys = [comm.all_reduce_rmsnorm(xs, ws, res, eps=1e-5, residual_out=p, mode="flash") for p in pre]
    assert comm.last_call()["kernel"] == "flash"
    comm.sync()
    for r in range(W):
        row = total(xs) + res[r].double()
        ref = row * torch.rsqrt(row.pow(2).mean(-1, keepdim=True) + 1e-5) * ws[r].double()
        for y, p in zip(ys, pre):
            assert torch.equal(p[r].double(), row)
            torch.testing.assert_close(y[r].double(), ref, rtol=rtol, atol=1e-6)


# Row lengths by 16-byte vectors per thread of the norm kernel (128 / 129 / 1024 / 1025 / 2048 vectors), one that is no whole
# number of vectors, and one weight off a 16-byte boundary.
@pytest.mark.parametrize("dtype,hidden,off", [(BF16, 1024, 0), (BF16, 1032, 0), (F16, 8192, 0), (F32, 4100, 0), (F32, 8192, 0), (BF16, 1001, 0), (BF16, 1024, 1)])
def test_norm_beyond_the_one_shot_staging(comm, dtype, hidden, off):
    """Above the staging's size the sum comes first and a kernel per rank normalises its rows: 1 + world launches."""
    if comm.world == 1:
        pytest.skip("a group of one stages nothing")
    W, rtol = comm.world, {F32: 2e-6, F16: 2.0 ** -10, BF16: 2.0 ** -7}[dtype]
    rows = comm.layout()["flash_cap"] // (hidden * torch.empty(0, dtype=dtype).element_size()) + 3
    xs = [whole((rows, hidden), dtype, r) for r in range(W)]
    res, ws = [whole((rows, hidden), dtype, 50 + r) for r in range(W)], [whole((hidden,), dtype, 90 + r, off) for r in range(W)]
    pre, before = [torch.empty_like(x) for x in xs], comm.launches
    ys = comm.all_reduce_rmsnorm(xs, ws, res, eps=1e-5, residual_out=pre, mode="stream")
    assert comm.launches - before == 1 + W
    plain = comm.all_reduce_rmsnorm(xs, ws, None, eps=1e-5, mode="stream")
    comm.sync()
    pick = torch.tensor([0, 1, rows // 2, rows - 2, rows - 1], device="cuda")
    s = total([x[pick] for x in xs])
    for r in (0, W - 1):
        for got, row in ((ys[r], s + res[r][pick].double()), (plain[r], s)):
            ref = row * torch.rsqrt(row.pow(2).mean(-1, keepdim=True) + 1e-5) * ws[r].double()
            torch.testing.assert_close(got[pick].double(), ref, rtol=rtol, atol=1e-6)
        assert torch.equal(pre[r][pick].double(), s + res[r][pick].double())
        assert torch.equal(pre[r].float(), sum(x.float() for x in xs) + res[r].float())


# (One row length of each number of vectors per thread, and the two forms that the row kernel does not take.)
@pytest.mark.parametrize("dtype,hidden,off,launches", [(BF16, 1024, 0, 1), (F16, 8192, 0, 1), (F32, 4100, 0, 1), (F32, 8192, 0, 1), (BF16, 1001, 0, 2), (BF16, 1024, 1, 2)])
def test_norm_right_above_the_one_shot_staging(comm, dtype, hidden, off, launches):
    """One launch, like any larger size, and two passes only for rows that the row kernel does not take."""
    if comm.world == 1:
        pytest.skip("a group of one stages nothing")
    W, rtol = comm.world, {F32: 2e-6, F16: 2.0 ** -10, BF16: 2.0 ** -7}[dtype]
    rows = comm.layout()["flash_cap"] // (hidden * torch.empty(0, dtype=dtype).element_size()) + 3
    xs, res = [whole((rows, hidden), dtype, r) for r in range(W)], [whole((rows, hidden), dtype, 50 + r) for r in range(W)]
    ws, pre, before = [whole((hidden,), dtype, 90 + r, off) for r in range(W)], [torch.empty_like(x) for x in xs], comm.launches
    ys = comm.all_reduce_rmsnorm(xs, ws, res, eps=1e-5, residual_out=pre)
    assert comm.launches - before == (1 if launches == 1 else 1 + W)
    s = sum(x.float() for x in xs)
    for r in (0, W - 1):
        row = s + res[r].float()
        assert torch.equal(pre[r].float(), row)
        ref = row * torch.rsqrt(row.double().pow(2).mean(-1, keepdim=True) + 1e-5) * ws[r].double()
        torch.testing.assert_close(ys[r].double(), ref, rtol=rtol, atol=1e-6)


@pytest.mark.parametrize("dtype,hidden", [(BF16, 4096), (F16, 1000), (F32, 8192)])
def test_norm_far_beyond_the_one_shot_staging(comm, dtype, hidden):
    """One launch; two passes (one launch and one per rank) for calls whose outputs lie on one another, on inputs or off a boundary.  Whole-number
    inputs: the sums are the same in both, the norms differ by their roundings."""
    if comm.world == 1:
        pytest.skip("a group of one stages nothing")
    W, size, rtol = comm.world, torch.empty(0, dtype=dtype).element_size(), {F32: 2e-6, F16: 2.0 ** -10, BF16: 2.0 ** -7}[dtype]
    rows = (comm.layout()["flash_cap"] + (1 << 20)) // (hidden * size) + 1
    xs, res = [whole((rows, hidden), dtype, r) for r in range(W)], [whole((rows, hidden), dtype, 50 + r) for r in range(W)]
    ws = [whole((hidden,), dtype, 90 + r) for r in range(W)]
    s = sum(x.float() for x in xs)

    def check(ys, pre, launches, residual=res):
        for r in range(W):
            row = s + (residual[r].float() if residual else 0)
            if pre:
                assert torch.equal(pre[r].float(), row)
            ref = row * torch.rsqrt(row.double().pow(2).mean(-1, keepdim=True) + 1e-5) * ws[r].double()
            torch.testing.assert_close(ys[r].double(), ref, rtol=rtol, atol=1e-6)
        assert comm.launches - before == launches

    before, pre = comm.launches, [torch.empty_like(x) for x in xs]
    check(comm.all_reduce_rmsnorm(xs, ws, res, eps=1e-5, residual_out=pre), pre, 1)
    assert comm.last_call()["kernel"] == "local_norm"
    before = comm.launches
    check(comm.all_reduce_rmsnorm(xs, ws, None, eps=1e-5), None, 1, None)
    keep, before = [r.clone() for r in res], comm.launches
    check(comm.all_reduce_rmsnorm(xs, ws, keep, eps=1e-5, residual_out=keep), keep, 1)
    # Two passes: in place; one tensor for every rank's rows; a weight off a 16-byte boundary; a geometry of the caller's.
    own, before = [x.clone() for x in xs], comm.launches
    check(comm.all_reduce_rmsnorm(own, ws, res, eps=1e-5, out=own), None, 1 + W)
    one, before = torch.empty_like(xs[0]), comm.launches
    check(comm.all_reduce_rmsnorm(xs, ws, res[:1] * W, eps=1e-5, residual_out=[one] * W), [one] * W, 1 + W, res[:1] * W)
    ws, before = [whole((hidden,), dtype, 90 + r, 1) for r in range(W)], comm.launches
    check(comm.all_reduce_rmsnorm(xs, ws, res, eps=1e-5, residual_out=pre), pre, 1 + W)
    before = comm.launches
    check(comm.all_reduce_rmsnorm(xs, ws, res, eps=1e-5, residual_out=pre, mode="stream"), pre, 1 + W)


@pytest.mark.parametrize("hidden,off,mode", [(4096, 0, "auto"), (4096, 0, "stream"), (1001, 0, "auto"), (1024, 1, "auto")])
@pytest.mark.parametrize("extra", [-1, 1, 1 << 20])
def test_norm_of_residuals_that_outputs_lie_on(comm, hidden, off, mode, extra):
    """The residual is the one that the call was given, in one launch and in two passes: a rank's rows go to its own residual; the residual is
    updated in place; rows go to the next rank's residual; one tensor is every rank's residual and its update.  `extra`: bytes above the one-shot kernel's staging."""
    W = comm.world
    if W == 1 and extra > 0:
        pytest.skip("a group of one stages nothing")
    if extra < 0 and (hidden % 8 or off or mode != "auto"):
        pytest.skip("below the staging these are refused, or the multi-GPU kernel's")
    staging = comm.layout()["flash_cap"] if W > 1 else 4 << 20
    rows = (staging + extra) // (2 * hidden) + (extra > 0)
    xs = [whole((rows, hidden), BF16, r) for r in range(W)]
    res, ws = [whole((rows, hidden), BF16, 50 + r) for r in range(W)], [whole((hidden,), BF16, 90 + r, off) for r in range(W)]
    s = sum(x.float() for x in xs)

    def check(ys, residual):
        for r in range(W):
            row = s + residual[r].float()
            ref = row * torch.rsqrt(row.pow(2).mean(-1, keepdim=True) + 1e-5) * ws[r].float()
            torch.testing.assert_close(ys[r].float(), ref, rtol=2.0 ** -7, atol=1e-6)

    own = [r.clone() for r in res]
    pre = [torch.empty_like(r) for r in res]
    check(comm.all_reduce_rmsnorm(xs, ws, own, eps=1e-5, out=own, residual_out=pre, mode=mode), res)
    assert all(torch.equal(p.float(), s + r.float()) for p, r in zip(pre, res))
    if extra < 0 or W == 1:
        return
    own = [r.clone() for r in res]
    check(comm.all_reduce_rmsnorm(xs, ws, own, eps=1e-5, residual_out=own, mode=mode), res)
    assert all(torch.equal(o.float(), s + r.float()) for o, r in zip(own, res))
    own = [r.clone() for r in res]
    check(comm.all_reduce_rmsnorm(xs, ws, own, eps=1e-5, out=own[1:] + own[:1], mode=mode), res)
    one = res[0].clone()
    check(comm.all_reduce_rmsnorm(xs, ws, [one] * W, eps=1e-5, residual_out=[one] * W, mode=mode), res[:1] * W)
    assert torch.equal(one.float(), s + res[0].float())


def test_norm_of_more_rows_than_a_grid_has_ctas():
    """2^29 + 1 rows of one vector for eight ranks: more CTAs than a launch takes, so the sum comes first.  Input and output are one tensor for all ranks."""
    if torch.cuda.mem_get_info()[0] < 24 << 30:
        pytest.skip("needs 16 GiB")
    n, W = 1 << 29, 8
    tile = whole((8192, 8), BF16, 1)
    x, y, w = torch.empty((n + 1, 8), dtype=BF16, device="cuda"), torch.empty((n + 1, 8), dtype=BF16, device="cuda"), whole((8,), BF16, 2)
    x[:n].view(-1, 8192, 8).copy_(tile)
    x[n] = tile[5]
    with yali.Comm.emulated(W, device=0) as c:
        c.all_reduce_rmsnorm([x] * W, [w] * W, None, eps=1e-5, out=[y] * W)
        assert c.last_call()["kernel"] == "local_sum"
        c.sync()
    row = W * tile.float()
    want = row * torch.rsqrt(row.pow(2).mean(-1, keepdim=True) + 1e-5) * w.float()
    for first in (0, n // 2, n - 8192):
        torch.testing.assert_close(y[first:first + 8192].float(), want, rtol=2.0 ** -7, atol=1e-6)
    torch.testing.assert_close(y[n].float(), want[5], rtol=2.0 ** -7, atol=1e-6)


# (Few, some and many rows: the norm kernel's cuts; rows beyond the staging in one launch, and in two passes by vectors and by elements.)
@pytest.mark.parametrize("rows,hidden,mode", [(3, 4096, "auto"), (90, 4096, "auto"), (600, 2944, "auto"), (50, 8192, "auto"), (0, 4096, "auto"),
                                              (0, 4096, "stream"), (0, 1001, "auto")])
def test_norms_whose_ranks_share_an_output(comm, rows, hidden, mode):
    """One tensor as every rank's output holds the last rank's rows, one as every rank's updated residual the last rank's; rows win over residuals."""
    W = comm.world
    if W == 1:
        pytest.skip("one output")
    rows = rows or (comm.layout()["flash_cap"] + (1 << 20)) // (2 * hidden) + 1
    xs = [whole((rows, hidden), BF16, r) for r in range(W)]
    res, ws = [whole((rows, hidden), BF16, 50 + r) for r in range(W)], [whole((hidden,), BF16, 90 + r) for r in range(W)]
    pre = [sum(x.float() for x in xs) + r.float() for r in res]
    want = [p * torch.rsqrt(p.pow(2).mean(-1, keepdim=True) + 1e-5) * w.float() for p, w in zip(pre, ws)]
    for shared in ([0] * W, [r % 2 for r in range(W)]):
        outs, ros = ([torch.zeros_like(xs[0]) for _ in range(2)] for _ in range(2))
        last = {k: max(r for r in range(W) if shared[r] == k) for k in shared}
        kept = [torch.empty_like(x) for x in xs]
        comm.all_reduce_rmsnorm(xs, ws, res, eps=1e-5, out=[outs[k] for k in shared], residual_out=kept, mode=mode)
        assert all(torch.equal(k.float(), p) for k, p in zip(kept, pre))
        for k, r in last.items():
            torch.testing.assert_close(outs[k].float(), want[r], rtol=2.0 ** -7, atol=1e-6)
        ys = comm.all_reduce_rmsnorm(xs, ws, res, eps=1e-5, residual_out=[ros[k] for k in shared], mode=mode)
        for y, w in zip(ys, want):
            torch.testing.assert_close(y.float(), w, rtol=2.0 ** -7, atol=1e-6)
        assert all(torch.equal(ros[k].float(), pre[r]) for k, r in last.items())
        comm.all_reduce_rmsnorm(xs, ws, res, eps=1e-5, out=[outs[k] for k in shared], residual_out=[outs[k] for k in shared], mode=mode)
        for k, r in last.items():
            torch.testing.assert_close(outs[k].float(), want[r], rtol=2.0 ** -7, atol=1e-6)


@pytest.mark.parametrize("mode", ["auto", "stream"])
def test_norms_that_take_memory_for_a_call_replay_from_a_graph(comm, mode):
    """An output on the rank's own residual (in two passes read from a copy) and one output for every rank, captured in one graph and replayed."""
    W, hidden = comm.world, 4096
    if W == 1:
        pytest.skip("one output, and a group of one stages nothing")
    rows = (comm.layout()["flash_cap"] + (1 << 20)) // (2 * hidden) + 1
    xs = [whole((rows, hidden), BF16, r) for r in range(W)]
    res, ws = [whole((rows, hidden), BF16, 50 + r) for r in range(W)], [whole((hidden,), BF16, 90 + r) for r in range(W)]
    pre = [sum(x.float() for x in xs) + r.float() for r in res]
    want = [p * torch.rsqrt(p.pow(2).mean(-1, keepdim=True) + 1e-5) * w.float() for p, w in zip(pre, ws)]
    own, one = [r.clone() for r in res], torch.empty_like(res[0])

    def calls():
        comm.all_reduce_rmsnorm(xs, ws, own, eps=1e-5, out=own, mode=mode)
        comm.all_reduce_rmsnorm(xs, ws, res, eps=1e-5, out=[one] * W, mode=mode)

    calls()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls()
    for _ in range(2):
        for o, r in zip(own, res):
            o.copy_(r)
        one.zero_()
        graph.replay()
        torch.cuda.synchronize()
        for y, w in zip(own + [one], want + want[-1:]):
            torch.testing.assert_close(y.float(), w, rtol=2.0 ** -7, atol=1e-6)


@pytest.mark.parametrize("odd", ["x", "weight", "residual", "out", "residual_out"])
@pytest.mark.parametrize("mode", ["auto", "flash"])
def test_norm_refuses_tensors_off_a_16_byte_boundary(comm, odd, mode):
    """One rank's tensor starts at an odd element: an error of the call, before any launch."""
    W, rows, hidden = comm.world, 4, 1024
    off = {r: {odd: 1} if r == W - 1 else {} for r in range(W)}
    t = {k: [whole((rows, hidden) if k != "weight" else (hidden,), BF16, r, off[r].get(k, 0)) for r in range(W)]
         for k in ("x", "weight", "residual", "out", "residual_out")}
    before = comm.launches
    with pytest.raises(RuntimeError, match="16-byte aligned"):
        comm.all_reduce_rmsnorm(t["x"], t["weight"], t["residual"], out=t["out"], residual_out=t["residual_out"], mode=mode)
    assert comm.launches == before


def test_last_call_names_the_kernel_that_ran(comm):
    W = comm.world
    x, w = [whole((4, 1024), F32, r) for r in range(W)], [torch.ones(1024, device="cuda")] * W
    ran = lambda: comm.last_call()["kernel"]  # noqa: E731
    comm.all_reduce(x)
    assert ran() == "local_sum"
    comm.all_reduce_rmsnorm(x, w)
    assert ran() == "local_norm"
    shards = comm.reduce_scatter(x)
    assert ran() == ("local_reduce_scatter" if W > 1 else "local_sum")
    comm.all_gather(shards, 4096)
    assert ran() == ("local_all_gather" if W > 1 else "local_sum")
    comm.all_reduce_host([t.cpu().pin_memory() for t in x])
    assert ran() == "local_host_sum"
    comm.all_reduce(x, mode="flash")
    assert ran() == comm.last_call()["variant"] == "flash"
    comm.sync()


def test_halves_of_the_multi_gpu_kernel_on_request(comm, monkeypatch):
    if comm.world == 1:
        pytest.skip("a group of one has no halves")
    monkeypatch.setenv("YALI_KERNEL_MODE", "stream")
    n = 40001
    xs = [whole((n,), F32, r) for r in range(comm.world)]
    full = comm.all_gather(comm.reduce_scatter(xs), n)
    comm.sync()
    assert comm.last_call()["variant"] == "stream" and not comm.last_call()["flags"] & ONE_LAUNCH
    assert torch.equal(full[-1].double(), total(xs))


@pytest.mark.parametrize("dtype", [F32, F16, BF16])
@pytest.mark.parametrize("n", [1, 7, 8, 4097, 131072, 131075, 2000003])
def test_host_buffers_where_they_are(comm, dtype, n):
    """Pinned host memory, one kernel; the sizes sit around a 16-byte unit and the 64 x 256 threads of the grid.  Inputs change
    between calls: nothing of an earlier call may be read."""
    W = comm.world
    for off in (0, 1):
        src = [torch.empty(n + off, dtype=dtype, pin_memory=True)[off:] for _ in range(W)]
        dst = [torch.empty(n + off, dtype=dtype, pin_memory=True)[off:] for _ in range(W)]
        for step in range(3):
            for r in range(W):
                src[r].copy_(torch.randint(-8, 9, (n,), generator=torch.Generator().manual_seed(step * 100 + r)).to(dtype))
            before = comm.launches
            comm.all_reduce_host(src, dst, scale=0.5)
            torch.cuda.synchronize()
            assert comm.launches - before == 1 and comm.last_call()["flags"] & 1 << 10
            want = torch.stack([s.double() for s in src]).sum(0) * 0.5
            assert all(torch.equal(d.double(), want) for d in dst)
    comm.all_reduce_host(src, src)  # in place
    torch.cuda.synchronize()
    assert all(torch.equal(s.double(), want * 2) for s in src)
    with pytest.raises(ValueError):
        comm.all_reduce_host([torch.zeros(8) for _ in range(W)])


def test_any_iterable_of_tensors_will_do(comm):
    """One tensor per rank from a generator, a tuple or a dict's values, for every argument of every call."""
    W = comm.world
    it = lambda ts: (t for t in ts)  # noqa: E731
    x, y = [whole((4, 128), BF16, r) for r in range(W)], [torch.empty(4, 128, dtype=BF16, device="cuda") for _ in range(W)]
    w, res = [torch.ones(128, dtype=BF16, device="cuda") for _ in range(W)], [whole((4, 128), BF16, 9) for _ in range(W)]
    for out in (None, y):
        got = comm.all_reduce(it(x), None if out is None else it(out))
        assert all(torch.equal(t.double(), total(x)) for t in got)
        assert out is None or all(t is o for t, o in zip(got, out))
        pre = [torch.empty_like(t) for t in x]
        got = comm.all_reduce_rmsnorm(it(x), tuple(w), it(res), out=out and it(out), residual_out=it(pre))
        assert len(got) == W and all(torch.equal(p.double(), total(x) + r.double()) for p, r in zip(pre, res))
        full = comm.all_gather(it(comm.reduce_scatter(it(x))), 512, None if out is None else it(out))
        assert all(torch.equal(t.double().view(4, 128), total(x)) for t in full)
        if W > 1:
            k = [torch.eye(128, dtype=BF16, device="cuda") for _ in range(W)]
            got = comm.fused_linear_rmsnorm(it(x), dict(enumerate(k)).values(), it(w), it(res), out=out and it(out), residual_out=it(pre))
            assert len(got) == W and all(torch.equal(p.double(), total(x) + r.double()) for p, r in zip(pre, res))
            assert out is None or all(t is o for t, o in zip(got, out))
    src, dst = [t.cpu().pin_memory() for t in x], [t.cpu().pin_memory() for t in y]
    for out in (None, dst):
        got = comm.all_reduce_host(it(src), out and it(out))
        torch.cuda.synchronize()
        assert len(got) == W and all(torch.equal(t.double(), total(src)) for t in got)
    comm.sync()


def test_arguments_of_the_wrong_type_are_type_errors(comm):
    x, w = [whole((4, 128), BF16, r) for r in range(comm.world)], [torch.ones(128, dtype=BF16, device="cuda")] * comm.world
    host = [t.cpu().pin_memory() for t in x]
    before = comm.launches
    for call in (lambda: comm.all_reduce(x, mode=None), lambda: comm.all_reduce(x, mode=3), lambda: comm.all_reduce(x, scale="2"),
                 lambda: comm.all_reduce(x, out_dtype="fp32"), lambda: comm.all_reduce(3), lambda: comm.all_reduce(["x"] * comm.world),
                 lambda: comm.all_reduce_rmsnorm(x, w, mode=None), lambda: comm.all_reduce_rmsnorm(x, w, eps="1"),
                 lambda: comm.all_reduce_host(host, mode=None), lambda: comm.all_reduce_host(host, scale=x),
                 lambda: comm.all_gather(x, "9")):
        with pytest.raises(TypeError):
            call()
    with pytest.raises(RuntimeError, match="negative"):
        comm.all_gather(x, -1)
    assert comm.launches == before
    y = [torch.empty_like(t) for t in x]
    assert comm.all_reduce(x, y, out_dtype="not looked at")[0] is y[0]
    comm.sync()


@pytest.mark.parametrize("which", ["src", "dst"])
def test_host_buffers_that_are_registered_in_part(which):
    """The first half of one buffer is registered, so it passes for pinned memory: the kernel must not be given it."""
    cudart, n = torch.cuda.cudart(), 1 << 20
    with yali.Comm.emulated(2, device=0) as c:
        part = torch.frombuffer(mmap.mmap(-1, n * 4), dtype=torch.float32).fill_(1)
        bufs = {k: [torch.ones(n).pin_memory() for _ in range(2)] for k in ("src", "dst")}
        bufs[which][1] = part
        assert int(cudart.cudaHostRegister(part.data_ptr(), n * 2, 0)) == 0
        try:
            assert part.is_pinned()
            try:
                c.all_reduce_host(bufs["src"], bufs["dst"])
            except RuntimeError:
                pass  # the copies may refuse it
            torch.cuda.synchronize()
            assert not c.last_call()["flags"] & 1 << 10
        finally:
            assert int(cudart.cudaHostUnregister(part.data_ptr())) == 0
        ok = [torch.ones(n).pin_memory() for _ in range(2)]
        assert torch.equal((c.all_reduce_host(ok), torch.cuda.synchronize())[0][1], torch.full((n,), 2.0))


@pytest.mark.parametrize("dtype", [F32, F16, BF16])
@pytest.mark.parametrize("n", [8, 16, 4099, 40001, 500000, 1 << 20])
def test_a_geometry_of_the_caller_runs_the_multi_gpu_kernels(comm, n, dtype):
    """`ctas` and `slot_bytes` without a mode: accepted by every collective, and nothing of them is dropped."""
    W = comm.world
    if W == 1:
        pytest.skip("a group of one has the one-shot kernel only")
    xs = [whole((n,), dtype, n + r) for r in range(W)]
    for kw in ({"ctas": 4}, {"slot_bytes": 2048}, {"ctas": 3, "slot_bytes": 4096}):
        ys = comm.all_reduce(xs, **kw)
        assert not comm.last_call()["flags"] & ONE_LAUNCH
        full = comm.all_gather(comm.reduce_scatter(xs, **kw), n, **kw)
        last = comm.last_call()
        assert last["variant"] == "stream" and last["ctas"] <= kw.get("ctas", 1 << 30)
        assert last["slot_bytes"] == kw.get("slot_bytes", last["slot_bytes"])
        comm.sync()
        assert all(torch.equal(t.double(), total(xs)) for t in ys + full)
    x, w = [t[:8].view(1, 8) for t in xs], [torch.ones(8, dtype=dtype, device="cuda")] * W
    y = comm.all_reduce_rmsnorm(x, w, ctas=1)
    assert not comm.last_call()["flags"] & ONE_LAUNCH
    comm.sync()
    row = total(x)
    # One rounding to the output type on top of the fp32 sum of squares and product.
    rtol = {F32: 2e-6, F16: 2.0 ** -10, BF16: 2.0 ** -7}[dtype]
    torch.testing.assert_close(y[0].double(), row * torch.rsqrt(row.pow(2).mean(-1, keepdim=True) + 1e-5), rtol=rtol, atol=1e-6)


@pytest.mark.parametrize("row_world", [2, 4])
def test_calls_with_a_tuning_table(tmp_path, row_world):
    """A table for the group names the kernel, on the device and for pinned host memory; one for another group changes nothing."""
    table = tmp_path / "table.json"
    table.write_text(json.dumps({"rows": [{"world": row_world, "elem_bytes": 4, "max_bytes": 1 << 40, "variant": "stream",
                                           "ctas": 8, "slot_bytes": 4096}]}))
    code = ("import torch, yali_b200 as yali\n"
            "c = yali.Comm.emulated(2, device=0)\n"
            "s = [torch.full((5000,), r + 1.0).pin_memory() for r in range(2)]\n"
            "d = c.all_reduce_host(s)\n"
            "torch.cuda.synchronize(); c.check()\n"
            "assert all(torch.equal(t, torch.full_like(t, 3.0)) for t in d)\n"
            "l = c.last_call(); print(l['variant'], bool(l['flags'] & 1 << 9))\n"
            "d = c.all_reduce([t.cuda() for t in s])\n"
            "c.sync(); assert all(torch.equal(t, torch.full_like(t, 3.0)) for t in d)\n"
            "l = c.last_call(); print(l['variant'], bool(l['flags'] & 1 << 9))\n")
    p = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, YALI_TUNING_FILE=str(table)), capture_output=True,
                       text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    assert p.stdout.split() == 2 * (["stream", "False"] if row_world == 2 else ["flash", "True"])


@pytest.mark.parametrize("n", [1, 255, 256, 257, 524288, 524289])
def test_new_outputs_of_one_call_are_apart(comm, n):
    """Outputs that the call makes (one allocation up to 4 MiB, else one per rank; 524288 elements of 2 bytes x 4 ranks is the
    line): contiguous, aligned, and writing one leaves the others and a later call's alone."""
    W = comm.world
    x = [torch.full((n,), r + 1.0, dtype=BF16, device="cuda") for r in range(W)]
    want = float(W * (W + 1) // 2)
    first, second = comm.all_reduce(x), comm.all_reduce(x, scale=2.0)
    first[0].fill_(-7.0)
    assert all(torch.equal(t, torch.full_like(t, want)) for t in first[1:])
    assert all(torch.equal(t, torch.full_like(t, 2 * want)) for t in second)
    assert all(t.shape == x[0].shape and t.is_contiguous() and t.data_ptr() % 16 == 0 for t in first + second)
