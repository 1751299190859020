"""Sums over blocks (loss sums, column sums), which the last block to arrive adds up or a second launch: one block, a few, all of
them; the counters serve the next call, of another size, as they did the first."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from ferrograd_b200 import GpuContext
    c = GpuContext(0)
    yield c
    c.sync()
    c.destroy()


def test_loss_sums(ctx):
    r = np.random.Generator(np.random.Philox(3))
    for n in (1, 255, 1025, 4096, 300007, 5, 2000003, 1024):
        p, t = r.random(n, np.float32) * 0.8 + 0.1, r.random(n, np.float32)
        pd, td, out, loss = ctx.init_tensor_f32((n,), p), ctx.init_tensor_f32((n,), t), ctx.new_tensor((1,)), ctx.new_tensor((n,))
        for again in range(2):
            ctx.mse_loss_grad(pd, td, n, loss_elem=loss, loss_sum=out)
            want = ((p.astype(np.float64) - t) ** 2).sum()
            # chains of at most 30 additions: 1e-5 is above 30 * 2^-24 and the roundings of the squares
            assert abs(ctx.to_numpy(out)[0] - want) <= 1e-5 * want
            ctx._check(ctx.lib.fg_sum_f32(ctx.handle, pd.ptr, n, out.ptr))
            want = p.astype(np.float64).sum()
            assert abs(ctx.to_numpy(out)[0] - want) <= 1e-5 * want


@pytest.mark.parametrize("M,N", [(1, 20), (255, 33), (257, 32), (512, 31), (513, 1000), (5000, 10), (4096, 64), (300, 40000)])
def test_column_sums(ctx, M, N):
    r = np.random.Generator(np.random.Philox(M + N))
    K = 4      # the exact path, whose bias gradient is a pass of its own
    dY, A = r.standard_normal((M, N), np.float32), r.standard_normal((M, K), np.float32)
    db, dB = ctx.new_tensor((N,)), ctx.new_tensor((K, N))
    dyd, ad = ctx.init_tensor_f32((M, N), dY), ctx.init_tensor_f32((M, K), A)
    for again in range(2):
        ctx.gemm_bwd(ad, None, dyd, M, N, K, dB=dB, dbias=db, mode="simt")
        want = dY.astype(np.float64).sum(0)
        # chains of at most 32 + 8 additions of partial sums below 4 sqrt(M): far below 1e-5 sqrt(M)
        assert np.abs(ctx.to_numpy(db) - want).max() <= 1e-5 * np.sqrt(M)


def test_cross_entropy_sums(ctx):
    # the loss dispatch of a graph that ends in softmax: one row to more elements than all blocks hold at once
    from ferrograd_b200.mlp import GraphMLP
    r = np.random.Generator(np.random.Philox(4))
    for rows, cols in ((1, 5), (64, 10), (33, 1000), (2500, 1001), (7, 3)):
        net = GraphMLP(ctx, [4, cols], rows, "gelu", "ce", ("sgd", 1e-3))
        net.set_params([r.standard_normal((4, cols), np.float32)], [r.standard_normal(cols, np.float32)])
        t = r.integers(0, cols, rows).astype(np.uint32)
        net.upload_batch(r.standard_normal((rows, 4), np.float32), t)
        for again in range(2):
            ctx.dispatch_forward(net.schedule)
            ctx.dispatch_loss(net.schedule, net.target)
            p = net.get_output().astype(np.float64)
            want = -np.log(p[np.arange(rows), t]).sum()
            # positive terms in at most 9 + 5 + 8 + 5 + 5 + 8 additions, and the logarithm's own roundings
            assert abs(net.get_loss() - want) <= 45 * 2.0 ** -24 * want, (rows, cols)
        net.destroy()


@pytest.mark.parametrize("n,called,recorded", [(1000, 1, 1), (100_001, 1, 2), (3_000_003, 2, 2)])
def test_sums_in_one_launch_or_two(ctx, n, called, recorded):
    # one block has the sum; a few are added by the last of them where the call's launches cost more, and by a second launch in a
    # plan; many by a second launch.  The same additions every time.
    r = np.random.Generator(np.random.Philox(n))
    p, t = ctx.init_tensor_f32((n,), r.random(n, np.float32) * 0.8 + 0.1), ctx.init_tensor_f32((n,), r.random(n, np.float32))
    outs = [ctx.new_tensor((1,)) for _ in range(3)]
    calls = [lambda: ctx.mse_loss_grad(p, t, n, loss_sum=outs[0]), lambda: ctx.bce_loss_grad(p, t, n, loss_sum=outs[1]),
             lambda: ctx._check(ctx.lib.fg_sum_f32(ctx.handle, p.ptr, n, outs[2].ptr))]
    for call, out in zip(calls, outs):
        before = ctx.launch_count()
        call()
        assert ctx.launch_count() - before == called
        first = ctx.to_numpy(out)[0]
        ctx.plan_begin()
        call()
        plan = ctx.plan_end()
        for again in range(2):
            ctx.memset_zero(out)
            before = ctx.launch_count()
            plan.launch()
            assert ctx.launch_count() - before == recorded
            assert ctx.to_numpy(out)[0] == first
        plan.destroy()


@pytest.mark.parametrize("M,N,called,recorded", [(200, 1000, 1, 1), (300, 1000, 1, 2), (3000, 40, 1, 2), (9000, 300, 2, 2)])
def test_column_sums_in_one_launch_or_two(ctx, M, N, called, recorded):
    r = np.random.Generator(np.random.Philox(M + N))
    dY, db = ctx.init_tensor_f32((M, N), r.standard_normal((M, N), np.float32)), ctx.new_tensor((N,))
    call = lambda: ctx.gemm_bwd(None, None, dY, M, N, 1, dbias=db, mode="simt")             # noqa: E731
    before = ctx.launch_count()
    call()
    assert ctx.launch_count() - before == called
    first = ctx.to_numpy(db)
    ctx.plan_begin()
    call()
    plan = ctx.plan_end()
    ctx.memset_zero(db)
    before = ctx.launch_count()
    plan.launch()
    assert ctx.launch_count() - before == recorded
    assert np.array_equal(ctx.to_numpy(db), first)
    plan.destroy()
