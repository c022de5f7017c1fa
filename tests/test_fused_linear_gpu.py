"""The fused tensor-parallel layer: row-parallel GEMM on tcgen05/TMEM whose epilogue
pushes partial rows to their owner, then all-reduce + residual + RMSNorm, against a
plain PyTorch fp64 reference of the same layer.  Ranks are emulated on one GPU (one
cooperative launch runs all ranks' CTAs).  Shapes follow the Llama-3-8B o_proj with
tensor parallelism 8: K = 512 per rank, hidden 4096, T in {1, 16, 128, 2048}."""
import pytest
import torch

import yali_b200 as yali

pytestmark = pytest.mark.gpu


def make_layer(world, T, K, N, seed=0):
    g = torch.Generator(device="cpu").manual_seed(seed)
    xs = [torch.randn(T, K, generator=g).to(torch.bfloat16).cuda() for _ in range(world)]
    ws = [(torch.randn(N, K, generator=g) * 0.02).to(torch.bfloat16).cuda() for _ in range(world)]
    nw = (torch.rand(N, generator=g) + 0.5).to(torch.bfloat16).cuda()
    res = torch.randn(T, N, generator=g).to(torch.bfloat16).cuda()
    return xs, ws, nw, res


def reference(xs, ws, nw, res, eps=1e-5):
    # Partials are rounded to bf16 before the cross-rank sum, as in the unfused composition
    # (bf16 GEMM output, then all-reduce).
    acc = None
    for x, w in zip(xs, ws):
        p = (x.double().cpu() @ w.double().cpu().T).to(torch.bfloat16).double()
        acc = p if acc is None else acc + p
    return yali.reference.residual_rmsnorm(acc, nw.double().cpu(), None if res is None else res.double().cpu(), eps)


@pytest.fixture(scope="module", params=[2, 8])
def comm(request):
    c = yali.Comm.emulated(request.param, device=0, timeout_ms=3000)
    yield c
    c.close()


@pytest.mark.parametrize("T", [1, 16, 128, 300, 2048])
@pytest.mark.parametrize("oneshot", [True, False])
def test_fused_linear_matches_reference(comm, T, oneshot):
    K, N = 512, 4096
    if oneshot and T * N * 2 > comm.layout()["gemm_cap"]:
        pytest.skip("one-shot landing zone too small for this many rows")
    xs, ws, nw, res = make_layer(comm.world, T, K, N, seed=T)
    W = comm.world
    res_out = [torch.empty(T, N, dtype=torch.bfloat16, device="cuda") for _ in range(W)]
    outs = comm.fused_linear_rmsnorm(xs, ws, [nw] * W, [res] * W, eps=1e-5, residual_out=res_out, oneshot=oneshot)
    comm.sync()
    ref, pre = reference(xs, ws, nw, res)
    for o in outs:
        torch.testing.assert_close(o.double().cpu(), ref, rtol=3e-2, atol=3e-2)
    for q in range(W):
        torch.testing.assert_close(res_out[q].double().cpu(), pre, rtol=2e-2, atol=2e-2 * W)
    for o in outs[1:]:
        assert torch.equal(o, outs[0])


@pytest.mark.parametrize("T", [1, 2, 9, 16, 17, 31, 33, 64])
def test_few_token_form_matches_reference(comm, T):
    """T <= 64: 128 x 256 tiles split along K, partial rows to every rank as flag-in-data lines, every rank normalises all rows."""
    K, N = 512, 4096
    W = comm.world
    xs, ws, nw, res = make_layer(W, T, K, N, seed=100 + T)
    ref, pre = reference(xs, ws, nw, res)
    res_out = [torch.empty(T, N, dtype=torch.bfloat16, device="cuda") for _ in range(W)]
    results = []
    for it in range(5):  # back to back without synchronisation: the two landing parities alternate
        results.append(comm.fused_linear_rmsnorm(xs, ws, [nw] * W, [res] * W, eps=1e-5, residual_out=res_out, decode=True))
    comm.sync()
    for outs in results:
        for o in outs:
            torch.testing.assert_close(o.double().cpu(), ref, rtol=3e-2, atol=3e-2)
        for o in outs[1:]:
            assert torch.equal(o, outs[0])
    for q in range(W):
        torch.testing.assert_close(res_out[q].double().cpu(), pre, rtol=2e-2, atol=2e-2 * W)
    with pytest.raises(RuntimeError, match="at most"):
        big = make_layer(W, 65, K, N, seed=1)
        comm.fused_linear_rmsnorm(big[0], big[1], [big[2]] * W, None, decode=True)


def test_few_token_form_other_shapes_and_alternation(comm):
    W = comm.world
    for (T, K, N) in [(8, 64, 128), (40, 1024, 2048), (5, 192, 512)]:
        xs, ws, nw, _ = make_layer(W, T, K, N, seed=K + 1)
        ref, _ = reference(xs, ws, nw, None)
        results = []
        for it in range(6):  # alternate with the tile form (its counters and landing zone are separate)
            results.append(comm.fused_linear_rmsnorm(xs, ws, [nw] * W, None, decode=bool(it % 2 == 0)))
        comm.sync()
        for outs in results:
            for o in outs:
                torch.testing.assert_close(o.double().cpu(), ref, rtol=3e-2, atol=3e-2)


def test_fused_linear_back_to_back_and_other_shapes(comm):
    W = comm.world
    for (T, K, N) in [(64, 64, 128), (200, 1024, 2048), (33, 192, 512)]:
        xs, ws, nw, _ = make_layer(W, T, K, N, seed=K)
        ref, _ = reference(xs, ws, nw, None)
        results = []
        for it in range(6):
            results.append(comm.fused_linear_rmsnorm(xs, ws, [nw] * W, None, oneshot=bool(it % 2)))
        comm.sync()
        for outs in results:
            for o in outs:
                torch.testing.assert_close(o.double().cpu(), ref, rtol=3e-2, atol=3e-2)


def test_fused_linear_rejects_bad_shapes(comm):
    W = comm.world
    xs, ws, nw, _ = make_layer(W, 8, 96, 256, seed=1)  # K not a multiple of 64
    with pytest.raises(RuntimeError, match="multiple"):
        comm.fused_linear_rmsnorm(xs, ws, [nw] * W, None)
    xs, ws, nw, _ = make_layer(W, 8, 64, 200, seed=1)  # N not a multiple of 128
    with pytest.raises(RuntimeError, match="multiple"):
        comm.fused_linear_rmsnorm(xs, ws, [nw] * W, None)
    comm.sync()


@pytest.mark.parametrize("world", [2, 3, 8])
@pytest.mark.parametrize("T", [1, 31, 33, 65, 161, 256, 257, 513])
@pytest.mark.parametrize("K,N", [(64, 128), (64, 384), (192, 1024)])
def test_tile_form_at_the_edges_of_its_tiles(world, T, K, N):
    """Token tiles are multiples of 32 up to 256 rows, column tiles are two units of 128 (the second may lie beyond N),
    rows go to two groups of warps in turn.  Whole-number inputs: partial sums, their sum and the new residual are
    exact in bf16 (below 256), so the residual is compared bit by bit; the norm adds one rounding (2^-8)."""
    g = torch.Generator(device="cuda").manual_seed(T * N + world)
    with yali.Comm.emulated(world, device=0) as c:
        pick = lambda *s, p: ((torch.rand(s, generator=g, device="cuda") < p).float() * torch.randint(-1, 2, s, generator=g, device="cuda")).to(torch.bfloat16)
        xs, ws = [pick(T, K, p=0.5) for _ in range(world)], [pick(N, K, p=0.5) for _ in range(world)]
        nw, res = torch.full((N,), 0.5, dtype=torch.bfloat16, device="cuda"), pick(T, N, p=0.9)
        want = sum(x.double() @ w.double().T for x, w in zip(xs, ws)) + res.double()
        assert want.abs().max() < 256
        y = want * torch.rsqrt(want.pow(2).mean(-1, keepdim=True) + 1e-5) * 0.5
        for oneshot in (False, True):
            pre = [torch.empty_like(res) for _ in range(world)]
            outs = [c.fused_linear_rmsnorm(xs, ws, [nw] * world, [res] * world, residual_out=pre, oneshot=oneshot, decode=False) for _ in range(3)]
            c.sync()
            for p in pre:
                assert torch.equal(p.double(), want)
            for o in outs[0] + outs[2]:
                torch.testing.assert_close(o.double(), y, rtol=2.0 ** -8, atol=1e-6)


@pytest.mark.parametrize("world", [2, 3, 8])
@pytest.mark.parametrize("T", [1, 31, 32, 33, 65, 255, 257, 513])
@pytest.mark.parametrize("K,N", [(64, 128), (64, 384), (192, 2176), (512, 4096)])
def test_ranks_on_one_gpu_add_in_the_gemm(world, T, K, N):
    """Automatically chosen calls of emulated ranks: one GEMM over all ranks' K extents (two kernels, no exchange).  Token
    tiles are multiples of 32 up to 256 rows, column tiles are 256 wide, K may be split; each rank has a residual and
    norm weights of its own.  Whole-number inputs: all sums are exact in bf16 (below 256), so the residual is
    compared bit by bit; the norm adds one rounding (2^-8)."""
    g = torch.Generator(device="cuda").manual_seed(T * N + world)

    def pick(*shape, p):
        keep = torch.rand(shape, generator=g, device="cuda") < p
        return (keep * torch.randint(-1, 2, shape, generator=g, device="cuda")).to(torch.bfloat16)

    with yali.Comm.emulated(world, device=0) as c:
        xs, ws = [pick(T, K, p=0.4) for _ in range(world)], [pick(N, K, p=0.4) for _ in range(world)]
        nw = [torch.full((N,), 0.5 + r, dtype=torch.bfloat16, device="cuda") for r in range(world)]
        res = [pick(T, N, p=0.9) for _ in range(world)]
        total = sum(x.double() @ w.double().T for x, w in zip(xs, ws))
        assert total.abs().max() < 255
        for residuals in (res, None):
            pre = [torch.empty_like(r) for r in res]
            before = c.launches
            results = [c.fused_linear_rmsnorm(xs, ws, nw, residuals, residual_out=pre) for _ in range(3)]
            assert c.launches - before == 6
            c.sync()
            for r in range(world):
                want = total + (res[r].double() if residuals else 0)
                assert torch.equal(pre[r].double(), want)
                y = want * torch.rsqrt(want.pow(2).mean(-1, keepdim=True) + 1e-5) * nw[r].double()
                for outs in results:
                    torch.testing.assert_close(outs[r].double(), y, rtol=2.0 ** -8, atol=1e-6)
        # The residual stream updated in place; an output on another rank's residual takes the multi-GPU form.
        keep = [r.clone() for r in res]
        c.fused_linear_rmsnorm(xs, ws, nw, keep, residual_out=keep)
        assert all(torch.equal(k.double(), total + r.double()) for k, r in zip(keep, res))
        before = c.launches
        c.fused_linear_rmsnorm(xs, ws, nw, res, out=res[1:] + res[:1])
        c.sync()
        assert c.launches - before == 1


# Every way in which the row kernel shares out rows: one rank of a row per CTA (flag-in-data lines of few and of many CTAs, flags), two and four
# ranks, groups that the last ranks do not fill; row widths that fill their last warp and that do not, with one and with two vectors per
# thread.
@pytest.mark.parametrize("world,T,K,N", [(8, 3, 64, 2304), (8, 33, 128, 4096), (4, 40, 64, 640), (4, 36, 256, 384), (2, 100, 256, 3968),
                                         (4, 75, 128, 1024), (3, 120, 64, 768), (2, 300, 64, 512), (5, 130, 64, 1280), (3, 260, 64, 2048),
                                         (7, 200, 128, 1152), (8, 161, 64, 1664), (4, 1025, 64, 1152), (6, 100, 64, 2176), (7, 60, 512, 2176),
                                         (8, 150, 256, 3200), (4, 400, 64, 3200), (3, 450, 64, 2304)])
def test_rows_of_ranks_on_one_gpu(world, T, K, N):
    """Whole-number inputs as above: residuals bit by bit, the norm to one rounding.  Two calls, the second with other inputs."""
    g = torch.Generator(device="cuda").manual_seed(T * N + world)

    def pick(*shape, p):
        keep = torch.rand(shape, generator=g, device="cuda") < p
        return (keep * torch.randint(-1, 2, shape, generator=g, device="cuda")).to(torch.bfloat16)

    with yali.Comm.emulated(world, device=0) as c:
        ws, calls = [pick(N, K, p=0.3) for _ in range(world)], []
        nw = [(torch.rand(N, generator=g, device="cuda") + 0.5).to(torch.bfloat16) for _ in range(world)]
        for _ in range(2):
            xs, res = [pick(T, K, p=0.3) for _ in range(world)], [pick(T, N, p=0.9) for _ in range(world)]
            pre, before = [torch.empty_like(r) for r in res], c.launches
            calls.append((xs, res, pre, c.fused_linear_rmsnorm(xs, ws, nw, res, residual_out=pre)))
            assert c.launches - before == 2
        c.sync()
        for xs, res, pre, outs in calls:
            total = sum(x.double() @ w.double().T for x, w in zip(xs, ws))
            assert total.abs().max() < 255
            for r in range(world):
                want = total + res[r].double()
                assert torch.equal(pre[r].double(), want)
                y = want * torch.rsqrt(want.pow(2).mean(-1, keepdim=True) + 1e-5) * nw[r].double()
                torch.testing.assert_close(outs[r].double(), y, rtol=2.0 ** -8, atol=1e-6)


@pytest.mark.parametrize("world", [2, 8])
def test_few_rows_back_to_back_with_new_inputs(world):
    """Sums as flag-in-data lines: 60 calls in one graph, rows and inputs changing from call to call, replayed three times.
    Whole-number inputs, so every call's residual is exact; one call's lines in another's result would show."""
    K, N = 512, 4096
    g = torch.Generator(device="cuda").manual_seed(world)

    def pick(*shape):
        keep = torch.rand(shape, generator=g, device="cuda") < 0.3
        return (keep * torch.randint(-1, 2, shape, generator=g, device="cuda")).to(torch.bfloat16)

    ws, nw = [pick(N, K) for _ in range(world)], [torch.ones(N, dtype=torch.bfloat16, device="cuda")] * world
    calls = []
    for i in range(60):
        T = (1, 8, 64, 3, 33)[i % 5]
        xs = [pick(T, K) for _ in range(world)]
        calls.append((xs, [torch.empty(T, N, dtype=torch.bfloat16, device="cuda") for _ in range(world)]))
    with yali.Comm.emulated(world, device=0, timeout_ms=2000) as c:
        c.fused_linear_rmsnorm(calls[0][0], ws, nw, None, residual_out=calls[0][1])
        c.sync()
        graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=side):
            for xs, pre in calls:
                c.fused_linear_rmsnorm(xs, ws, nw, None, residual_out=pre)
        for _ in range(3):
            for _xs, pre in calls:
                for p in pre:
                    p.zero_()
            graph.replay()
            torch.cuda.synchronize()
            c.check()
            for xs, pre in calls:
                want = sum(x.double() @ w.double().T for x, w in zip(xs, ws))
                assert want.abs().max() < 256
                assert all(torch.equal(p.double(), want) for p in pre)
        del graph
