"""The narrow layer's backward kernels at few samples, where chunks shrink and a single chunk takes the exact path (of a long k: the FMA
kernel takes the smaller layers), the line between the two, and the multi-tensor update at the sizes where its chunks shrink."""
import numpy as np
import pytest

from conftest import rel_err_ok

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from ferrograd_b200 import GpuContext
    c = GpuContext(0)
    yield c
    c.sync()
    c.destroy()


def check(x, ref, what):
    # sums of at most 1100 f32 products in chunks of 16 to 64: 2^-24 * sqrt(1100) * 5 with the reference's own error on top
    ok, worst = rel_err_ok(x, ref, 2e-5)
    assert ok, f"{what}: {worst:.3g}"


@pytest.mark.parametrize("M,N,K", [(1, 2, 16), (8, 16, 5), (64, 16, 2), (65, 10, 33), (100, 4, 520), (384, 12, 256), (1100, 3, 64), (64, 1, 8193), (50, 2, 20001),
                                   (8, 16, 50_000), (64, 16, 4100), (65, 13, 5100), (100, 4, 10_600), (384, 12, 920), (1100, 3, 1300)])
def test_backward(ctx, oracle, M, N, K):
    r = np.random.Generator(np.random.Philox(M + N + K))
    f = lambda *s: r.standard_normal(s).astype(np.float32)                    # noqa: E731
    up = lambda a: ctx.init_tensor_f32(a.shape, a)                            # noqa: E731
    A, B, dZ, saved = f(M, K), f(K, N), f(M, N), np.tanh(f(M, K))
    dB, dA, db, db_below = (ctx.new_tensor(s) for s in ((K, N), (M, K), (N,), (K,)))
    sa = (M * K + 7) // 8 * 8
    ctx.gemm_bwd_paired(up(A), up(B), up(dZ), M, N, K, dB=dB, dbias=db, dA=dA, below_act="tanh", below_saved=up(saved),
                        dA_pairs=ctx.alloc_zeroed(4 * sa), dA_stride=sa, below_dbias=db_below)
    ref = oracle.act_bwd(oracle.gemm(dZ, B, transB=True, f64=True), saved, "tanh")
    check(ctx.to_numpy(dB), oracle.gemm(A, dZ, transA=True, f64=True), "dB")
    check(ctx.to_numpy(dA), ref, "dA")
    check(ctx.to_numpy(db), dZ.astype(np.float64).sum(0), "dbias")
    check(ctx.to_numpy(db_below), ref.astype(np.float64).sum(0), "bias gradient of the layer below")


@pytest.mark.parametrize("sizes", [(1,), (1023, 1025), (5000, 0, 3), (700_001, 17), tuple([300] * 15 + [0] + [500] * 4)])
def test_update_of_several_tensors(ctx, oracle, sizes):
    r = np.random.Generator(np.random.Philox(len(sizes)))
    w, g = [r.standard_normal(n).astype(np.float32) for n in sizes], [r.standard_normal(n).astype(np.float32) for n in sizes]
    place = lambda a: ctx.init_tensor_f32((max(a.size, 1),), a if a.size else np.zeros(1, np.float32))       # noqa: E731
    wd, gd = [place(a) for a in w], [place(a) for a in g]
    ctx.sgd_step_multi([dict(w=a, g=b, n=n) for a, b, n in zip(wd, gd, sizes)], 0.1)
    for a, b, n, dw, dg in zip(w, g, sizes, wd, gd):
        if n:
            oracle.sgd(a, b, 0.1)
            assert np.array_equal(ctx.to_numpy(dw), a) and (ctx.to_numpy(dg) == 0).all()


# Small products of a narrow layer: the FMA kernel for few rows, the kernels above for many; either side of the lines between them (rows, and
# rows x inputs; with the layer below, without, with an activation of its own), which kernels ran by the timing records.
@pytest.mark.parametrize("M,N,K,narrow", [(3072, 3, 2, (False, True, True)), (3073, 3, 2, (True, True, True)), (3072, 4, 2, (False, False, True)),
                                          (3073, 4, 2, (True, True, True)), (2048, 3, 5, (False, False, True)), (2049, 3, 5, (False, True, True)),
                                          (1024, 1, 97, (False, False, False)), (1024, 1, 98, (False, False, True)), (4096, 16, 3, (False, False, True)),
                                          (4097, 16, 3, (True, True, True)), (2048, 16, 60, (False, False, False)), (2049, 16, 60, (False, False, True)),
                                          (1000, 4, 205, (False, False, True)), (1000, 4, 206, (True, True, True)), (64, 1, 4007, (False, False, True)),
                                          (64, 1, 4008, (True, True, True)), (60_001, 10, 6, (True, True, True)), (20, 16, 19_000, (True, True, True))])
def test_few_rows_and_many(ctx, oracle, M, N, K, narrow):
    r = np.random.Generator(np.random.Philox(M + N + K))
    f = lambda *s: r.standard_normal(s).astype(np.float32)                    # noqa: E731
    up = lambda a: ctx.init_tensor_f32(a.shape, a)                            # noqa: E731
    A, B, dY, S, S1 = f(M, K), f(K, N), f(M, N), np.tanh(f(M, N)), np.tanh(f(M, K))
    a, b, y, s, s1 = (up(x) for x in (A, B, dY, S, S1))
    dz = oracle.act_bwd(dY, S, "tanh")
    out = lambda: [up(np.full(sh, np.nan, np.float32)) for sh in ((M, K), (K, N), (N,), (K,))]      # noqa: E731
    # sums of k products in chains of at most k: 2^-24 * sqrt(k), five deviations of it, and 16 roundings of 2^-24 for the factor 1 - s * s and
    # its product (three) and the oracle's own in f32
    close = lambda x, ref, k, what: rel_err_ok(ctx.to_numpy(x), ref, 2.0 ** -24 * (16 + 5 * k ** 0.5))[0] or pytest.fail(what)      # noqa: E731

    def ran(call):
        ctx.timing_enable(True)
        call()
        n = ctx.timing_read("skinny")[0]
        ctx.timing_enable(False)
        return n > 0

    dA, dB, db, below = out()
    assert ran(lambda: ctx.gemm_bwd_paired(a, b, y, M, N, K, dB=dB, dbias=db, dA=dA, below_act="tanh", below_saved=s1, below_dbias=below)) == narrow[0]
    ref = oracle.act_bwd(oracle.gemm(dY, B, transB=True, f64=True), S1, "tanh")
    close(dA, ref, N, "dA below")
    close(dB, oracle.gemm(A, dY, transA=True, f64=True), M, "dB below")
    close(db, dY.astype(np.float64).sum(0), M, "dbias below")
    close(below, ref.astype(np.float64).sum(0), M, "bias gradient of the layer below")
    for k, (z, kw) in enumerate(((dY, dict(act="none")), (dz, dict(act="tanh", saved=s)))):
        dA, dB, db, _ = out()
        assert ran(lambda: ctx.gemm_bwd(a, b, y, M, N, K, dA=dA, dB=dB, dbias=db, **kw)) == narrow[1 + k]
        close(dA, oracle.gemm(z, B, transB=True, f64=True), N, "dA")
        close(dB, oracle.gemm(A, z, transA=True, f64=True), M, "dB")
        alone = out()[0]
        ctx.gemm_bwd(None, b, y, M, N, K, dA=alone, **kw)
        close(alone, oracle.gemm(z, B, transB=True, f64=True), N, "dA alone")
        close(db, z.astype(np.float64).sum(0), M, "dbias")


def test_many_rows_are_recorded_in_the_room_for_dz(oracle):
    # 5000 rows are the narrow layer's kernels', but not where a recording's arena has room for dZ alone
    from ferrograd_b200 import GpuContext
    M, N, K = 5000, 2, 4
    c = GpuContext(0)
    c.reserve_workspace(M * N * 4 + (M + 255) // 256 * N * 4 + 1024)
    r = np.random.Generator(np.random.Philox(8))
    f = lambda *s: r.standard_normal(s).astype(np.float32)                    # noqa: E731
    A, B, dY, S = f(M, K), f(K, N), f(M, N), np.tanh(f(M, N))
    t = [c.init_tensor_f32(x.shape, x) for x in (A, B, dY, S)]
    dA, dB, db = (c.new_tensor(s) for s in ((M, K), (K, N), (N,)))
    c.plan_begin()
    c.gemm_bwd(t[0], t[1], t[2], M, N, K, act="tanh", saved=t[3], dA=dA, dB=dB, dbias=db)
    plan = c.plan_end()
    plan.launch()
    dz = oracle.act_bwd(dY, S, "tanh")
    close = lambda x, ref, what: rel_err_ok(c.to_numpy(x), ref, 2.0 ** -24 * (16 + 5 * M ** 0.5))[0] or pytest.fail(what)      # noqa: E731
    close(dA, oracle.gemm(dz, B, transB=True, f64=True), "dA")
    close(dB, oracle.gemm(A, dz, transA=True, f64=True), "dB")
    close(db, dz.astype(np.float64).sum(0), "dbias")
    plan.destroy()
    c.destroy()
