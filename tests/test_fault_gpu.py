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
