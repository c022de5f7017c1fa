"""Failure detection on the device without faulting it: one rank's kernel leaves at
once (as if that rank had never launched), so the flags its peers wait for are never
set.  Their waits must run out after the communicator's limit, the kernel must
return normally, the host must see a Timeout with the place of the wait, and after
reset() the communicator must work again."""
import pytest
import torch

import yali_b200 as yali
from yali_b200 import _native
from yali_b200.parallel.comm import YaliTimeout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["flash", "stream"])
@pytest.mark.parametrize("world", [2, 4])
def test_wait_runs_out_then_reset_recovers(mode, world):
    ext = _native.ext()
    with yali.Comm.emulated(world, device=0, timeout_ms=150) as comm:
        xs = []
        for r in range(world):
            t = torch.empty(40000, dtype=torch.float32, device="cuda:0")
            ext.fill_random(t, 0, 1234 + r)
            xs.append(t)
        comm.all_reduce(xs, mode=mode)  # healthy call first
        comm.sync()
        comm.all_reduce(xs, mode=mode, _skip_rank=1)
        with pytest.raises(YaliTimeout) as info:
            comm.sync()
        assert "waiting for rank 1" in str(info.value)
        assert "waiting for rank 1" in comm.status()
        with pytest.raises(YaliTimeout):  # poisoned until reset
            comm.all_reduce(xs, mode=mode)
        comm.reset()
        assert comm.status() == ""
        outs = comm.all_reduce(xs, mode=mode)
        comm.sync()
        for o in outs:
            assert ext.validate_sum(o, torch.float32, 0, 1234, world)["mismatches"] == 0
        # the GPU context is intact
        assert torch.ones(4, device="cuda:0").sum().item() == 4.0


@pytest.mark.parametrize("world", [2, 8])
def test_reset_forgets_the_flag_in_data_lines(world):
    """After reset() call numbers start again, so what the calls before it left in the staging must not pass for this
    call's data: the small one-shot, and a rank of it that never launches."""
    with yali.Comm.emulated(world, device=0, timeout_ms=150) as comm:
        xs = [torch.full((4096,), float(r), device="cuda:0") for r in range(world)]
        comm.all_reduce(xs, mode="flash")
        comm.sync()
        assert comm.last_call()["flags"] & 64  # flag in data
        comm.reset()
        ys = [x + 1 for x in xs]
        comm.all_reduce(ys, mode="flash", _skip_rank=1)
        with pytest.raises(YaliTimeout):
            comm.sync()
        comm.reset()
        outs = comm.all_reduce(ys, mode="flash")
        comm.sync()
        want = float(world * (world - 1) // 2 + world)
        assert all(torch.equal(o, torch.full_like(o, want)) for o in outs)


@pytest.mark.parametrize("world", [2, 8])
@pytest.mark.parametrize("form", [None, True])  # by size (ranks on one GPU add in the GEMM), few-token kernel
def test_fused_layer_of_few_rows_after_reset(world, form):
    K, N = 512, 4096
    with yali.Comm.emulated(world, device=0, timeout_ms=2000) as comm:
        g = torch.Generator(device="cuda:0").manual_seed(3)
        pick = lambda *s: torch.randint(-1, 2, s, generator=g, device="cuda:0").to(torch.bfloat16)  # noqa: E731
        w = torch.zeros(N, K, device="cuda:0", dtype=torch.bfloat16)
        w[:, 0] = 1  # every sum is the first column of x, added over the ranks: exact
        ws, nw = [w] * world, [torch.ones(N, dtype=torch.bfloat16, device="cuda:0")] * world
        for T in (8, 1, 33):
            for _ in range(3):
                xs, pre = [pick(T, K) for _ in range(world)], [torch.empty(T, N, dtype=torch.bfloat16, device="cuda:0") for _ in range(world)]
                comm.fused_linear_rmsnorm(xs, ws, nw, None, residual_out=pre, decode=form)
                comm.sync()
                want = sum(x[:, :1].double() for x in xs).expand(T, N)
                assert all(torch.equal(p.double(), want) for p in pre)
                comm.reset()


@pytest.mark.parametrize("form", [{}, {"oneshot": False}])
def test_time_limit_in_the_middle_of_a_fused_layer(form):
    """A call that takes longer than the limit: the GEMM's waits run out while its copies and MMAs are under way.  The call
    ends with an error, and what runs on the same SMs afterwards is right."""
    world = 8
    T, K, N = 4096, 16384, 4096  # 2.7 ms at the tensor cores' rate
    big_x, big_w = (torch.ones(n, K, dtype=torch.bfloat16, device="cuda:0") for n in (T, N))
    with yali.Comm.emulated(world, device=0, timeout_ms=1) as comm:
        for turn in range(3):
            nw = [torch.ones(N, dtype=torch.bfloat16, device="cuda:0")] * world
            comm.fused_linear_rmsnorm([big_x] * world, [big_w] * world, nw, None, **form)
            with pytest.raises(YaliTimeout):
                comm.sync()
            comm.reset()
            for k in (64, 1024):
                x = [torch.randint(-1, 2, (8, k), device="cuda:0").to(torch.bfloat16) for _ in range(world)]
                w = [torch.eye(N, k, dtype=torch.bfloat16, device="cuda:0")] * world
                pre = [torch.empty(8, N, dtype=torch.bfloat16, device="cuda:0") for _ in range(world)]
                comm.fused_linear_rmsnorm(x, w, nw, None, residual_out=pre, **form)
                comm.sync()
                want = torch.nn.functional.pad(sum(t.double() for t in x), (0, N - k))
                assert all(torch.equal(p.double(), want) for p in pre)


def test_time_limit_in_the_middle_of_a_pipelined_all_reduce():
    n = 1 << 29  # 8.6 GB in and out: 1.3 ms at least
    with yali.Comm.emulated(2, device=0, timeout_ms=1) as comm:
        xs = [torch.ones(n, device="cuda:0") for _ in range(2)]
        ys = [torch.empty_like(x) for x in xs]
        for turn in range(3):
            comm.all_reduce(xs, ys, mode="stream_direct")
            with pytest.raises(YaliTimeout):
                comm.sync()
            comm.reset()
            small = comm.all_reduce([x[:300000] for x in xs], mode="stream_direct")
            comm.sync()
            assert all(torch.equal(t, torch.full_like(t, 2.0)) for t in small)
