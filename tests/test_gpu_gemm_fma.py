"""Products with plain FMAs in shares of k (few samples, or few multiply-adds): sizes around the four tile heights (4, 16, 32, 64),
the tile's 64 columns, the stages' 32 and 64 k and the clusters' shares, in every orientation, on 16-byte boundaries and off them.  Among
them forward products of a short k, which are the exact path's."""
import math

import numpy as np
import pytest

from conftest import rel_err_ok

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from ferrograd_b200 import GpuContext
    c = GpuContext(0)
    yield c
    assert c.device_status() == 0
    c.destroy()


def rng(seed):
    return np.random.Generator(np.random.Philox(seed))


def up(ctx, a, shift=0):
    """The array on the device, `shift` words behind a 16-byte boundary; returns (owner, address)."""
    t = ctx.init_tensor_f32((a.size + shift,), np.concatenate([np.zeros(shift, np.float32), np.ascontiguousarray(a, np.float32).ravel()]))
    return t, t.ptr + 4 * shift


def check(x, ref, k, what):
    # a chain of k rounded additions of products, in the 2-norm's scale 2^-24 * sqrt(k), five deviations of it, and the activation's own
    ok, worst = rel_err_ok(x, ref, 2.0 ** -24 * (16 + 5 * math.sqrt(k)))
    assert ok, f"{what}: {worst:.3g}"


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (1, 64, 4096), (3, 65, 33), (4, 129, 200), (5, 63, 64), (16, 64, 2050), (17, 100, 31), (32, 16, 515),
                                   (33, 200, 96), (63, 1, 1000), (40, 288, 2016), (64, 64, 64), (100, 130, 65), (1, 4100, 36), (5, 63, 66), (3, 65, 97)])
@pytest.mark.parametrize("tA,tB", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("shift", [0, 1])
def test_forward(ctx, oracle, M, N, K, tA, tB, shift):
    r = rng(M * 7 + N * 3 + K)
    A, B = r.standard_normal((K, M) if tA else (M, K), np.float32), r.standard_normal((N, K) if tB else (K, N), np.float32)
    bias = r.standard_normal(N, np.float32)
    a, b, v = up(ctx, A, shift), up(ctx, B, shift), up(ctx, bias, shift)
    C, P = up(ctx, np.zeros((M, N)), shift), up(ctx, np.zeros((M, N)), shift)
    ctx.gemm(a[1], b[1], C[1], M, N, K, transA=tA, transB=tB, bias=v[1], act="tanh", preact_out=P[1])
    z = oracle.gemm(A, B, transA=tA, transB=tB, f64=True).astype(np.float64) + bias
    got = ctx.to_numpy(P[0])[shift:].reshape(M, N)
    check(got, z, K, "pre-activation")
    # of the stored sum: an error of z, which is sqrt(k) large, passes through tanh's slope of one onto an output of at most one
    check(ctx.to_numpy(C[0])[shift:].reshape(M, N), np.tanh(got.astype(np.float64)), 0, "output")


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (2, 70, 64), (32, 2050, 100), (50, 53, 960), (64, 2, 16), (63, 300, 7), (1544, 12, 37), (384, 10, 256), (100, 33, 65),
                                   (1000, 4, 4), (5, 128, 260)])
@pytest.mark.parametrize("act", ["none", "relu", "tanh", "gelu"])
@pytest.mark.parametrize("shift", [0, 3])
def test_backward(ctx, oracle, M, N, K, act, shift):
    r = rng(M + N * 5 + K * 3)
    f = lambda *s: r.standard_normal(s).astype(np.float32)                    # noqa: E731
    A, B, dY, S = f(M, K), f(K, N), f(M, N), np.tanh(f(M, N))
    t = [up(ctx, x, shift) for x in (A, B, dY, S)]
    empty = lambda: [up(ctx, np.full(s, np.nan), shift) for s in ((M, K), (K, N), (N,))]      # noqa: E731
    dz = oracle.act_bwd(dY, S, act) if act != "none" else dY
    refs = ((oracle.gemm(dz, B, transB=True, f64=True), N, "dA"), (oracle.gemm(A, dz, transA=True, f64=True), M, "dB"), (dz.astype(np.float64).sum(0), M, "dbias"))

    def same(outs, what, wanted=(True, True, True)):
        for o, (ref, k, name), wants in zip(outs, refs, wanted):
            x = ctx.to_numpy(o[0])[shift:].reshape(ref.shape)
            if wants:
                check(x, ref, k, what + name)
            else:
                assert np.isnan(x).all(), what + name + " was not asked for"

    sv = t[3][1] if act != "none" else None
    dA, dB, db = empty()
    ctx.gemm_bwd(t[0][1], t[1][1], t[2][1], M, N, K, act=act, saved=sv, dA=dA[1], dB=dB[1], dbias=db[1])
    same((dA, dB, db), "")
    # the gradients one by one, and the gradient of A over A itself
    dA, dB, db = empty()
    ctx.gemm_bwd(t[0][1], None, t[2][1], M, N, K, act=act, saved=sv, dB=dB[1])
    same((dA, dB, db), "one by one, ", (False, True, False))
    ctx.gemm_bwd(None, t[1][1], t[2][1], M, N, K, act=act, saved=sv, dA=dA[1], dbias=db[1])
    same((dA, dB, db), "one by one, ")
    _, dB, db = empty()
    ctx.gemm_bwd(t[0][1], t[1][1], t[2][1], M, N, K, act=act, saved=sv, dA=t[0][1], dB=dB[1], dbias=db[1])
    same((t[0], dB, db), "over A, ")


@pytest.mark.parametrize("M,N", [(40, 40), (8, 200)])
def test_gradients_over_what_dz_is_made_of(ctx, oracle, M, N):
    # dA over the saved tensor and dB over dY where the sizes agree: dZ is formed before either is written
    r = rng(M)
    f = lambda *s: r.standard_normal(s).astype(np.float32)                    # noqa: E731
    A, B, dY, S = f(M, N), f(N, N), f(M, N), f(M, N)
    a, b, y, sv = (up(ctx, x) for x in (A, B, dY, S))
    dz = oracle.act_bwd(dY, S, "gelu")
    dB = up(ctx, np.zeros((N, N)))
    ctx.gemm_bwd(a[1], b[1], y[1], M, N, N, act="gelu", saved=sv[1], dA=sv[1], dB=y[1] if M == N else dB[1])
    check(ctx.to_numpy(sv[0]).reshape(M, N), oracle.gemm(dz, B, transB=True, f64=True), N, "dA over the saved tensor")
    check(ctx.to_numpy(y[0] if M == N else dB[0]).reshape(N, N), oracle.gemm(A, dz, transA=True, f64=True), M, "dB")


@pytest.mark.parametrize("M,N,K", [(3, 20, 30), (16, 2, 64), (55, 60, 146), (128, 26, 32), (70, 100, 130), (300, 9, 21)])
@pytest.mark.parametrize("over", [False, True])
def test_paired_backward(ctx, oracle, M, N, K, over):
    # the factor of the layer below, the pairs and the column sums of dA, in the same launch; dA over the saved tensor
    r = rng(M * N)
    f = lambda *s: r.standard_normal(s).astype(np.float32)                    # noqa: E731
    A, B, dZ, S = f(M, K), f(K, N), f(M, N), f(M, K)
    a, b, z, sv = (up(ctx, x) for x in (A, B, dZ, S))
    dA = sv if over else up(ctx, np.zeros((M, K)))
    dB, db, below = (up(ctx, np.zeros(s)) for s in ((K, N), (N,), (K,)))
    stride = (M * K + 7) // 8 * 8
    pairs = ctx.new_tensor((2, stride), np.uint16)
    ctx.gemm_bwd_paired(a[1], b[1], z[1], M, N, K, dB=dB[1], dbias=db[1], dA=dA[1], below_act="gelu", below_saved=sv[1], dA_pairs=pairs,
                        dA_stride=stride, below_dbias=below[1])
    ref = oracle.act_bwd(oracle.gemm(dZ, B, transB=True, f64=True), S, "gelu")
    got = ctx.to_numpy(dA[0]).reshape(M, K)
    check(got, ref, N, "dA")
    check(ctx.to_numpy(dB[0]).reshape(K, N), oracle.gemm(A, dZ, transA=True, f64=True), M, "dB")
    check(ctx.to_numpy(db[0]), dZ.astype(np.float64).sum(0), M, "dbias")
    check(ctx.to_numpy(below[0]), got.astype(np.float64).sum(0), M, "bias gradient of the layer below")
    from ferrograd_b200.backend import to_bf16_bits
    hi = (got.view(np.uint32) & np.uint32(0xffffe000)).view(np.float32)
    p = ctx.to_numpy(pairs)[:, :M * K]
    assert np.array_equal(p[0], to_bf16_bits(got).ravel()) and np.array_equal(p[1], to_bf16_bits(got - hi).ravel())


# Around the most multiply-adds that this kernel takes: M * N * K, padded to its tiles, of 45 million forward and 32 or 40 million backward.
@pytest.mark.parametrize("M,N,K", [(384, 256, 416), (352, 250, 481), (352, 250, 512), (128, 17, 1600), (128, 25, 1900), (1000, 100, 161), (96, 3000, 36)])
@pytest.mark.parametrize("act", ["relu", "gelu"])
def test_both_sides_of_the_range(ctx, oracle, M, N, K, act):
    r = rng(M + N + K)
    f = lambda *s: r.standard_normal(s).astype(np.float32)                    # noqa: E731
    A, B, dY, S, bias = f(M, K), f(K, N), f(M, N), f(M, N), f(N)
    a, b, y, sv, v = (up(ctx, x) for x in (A, B, dY, S, bias))
    C, P = (up(ctx, np.full((M, N), np.nan)) for _ in range(2))
    # (the tensor-core kernels of the far side split an f32 into a tf32 and a bf16 rest: 2^-19 of a term)
    close = lambda x, ref, k, what: rel_err_ok(x, ref, 2.0 ** -24 * (16 + 5 * math.sqrt(k)) + 2.0 ** -19)[0] or pytest.fail(what)   # noqa: E731
    ctx.gemm(a[1], b[1], C[1], M, N, K, bias=v[1], act=act, preact_out=P[1])
    close(ctx.to_numpy(P[0]).reshape(M, N), oracle.gemm(A, B, f64=True) + bias, K, "pre-activation")
    dz = oracle.act_bwd(dY, S, act)
    refs = {"dA": (oracle.gemm(dz, B, transB=True, f64=True), N), "dB": (oracle.gemm(A, dz, transA=True, f64=True), M)}
    for grads in (("dA", "dB"), ("dB",), ("dA",)):
        out = {"dA": up(ctx, np.full((M, K), np.nan)), "dB": up(ctx, np.full((K, N), np.nan))}
        db = up(ctx, np.full(N, np.nan))
        ctx.gemm_bwd(a[1], b[1], y[1], M, N, K, act=act, saved=sv[1], dbias=db[1], **{g: out[g][1] for g in grads})
        for g, (ref, k) in refs.items():
            x = ctx.to_numpy(out[g][0]).reshape(ref.shape)
            if g in grads:
                close(x, ref, k, f"{g} of {grads}")
            else:
                assert np.isnan(x).all(), f"{g} of {grads}"
        close(ctx.to_numpy(db[0]), dz.astype(np.float64).sum(0), M, f"dbias of {grads}")


@pytest.mark.parametrize("T,M,N,K", [(1, 4, 4, 4), (7, 33, 66, 97), (24, 128, 26, 44), (3, 2, 300, 256), (9, 19, 335, 256), (31, 60, 500, 70)])
@pytest.mark.parametrize("act", ["none", "gelu"])
@pytest.mark.parametrize("gap", [0, 5])
def test_batched(ctx, oracle, T, M, N, K, act, gap):
    r = rng(T * M + N + K)
    f = lambda *s: r.standard_normal(s).astype(np.float32)                    # noqa: E731
    A, B, dY, S = f(T, M * K + gap), f(T, K * N + gap), f(T, M * N + gap), f(T, M * N + gap)
    a, b, y, sv = (up(ctx, x) for x in (A, B, dY, S))
    C, dA, dB = (up(ctx, np.zeros(x.shape)) for x in (dY, A, B))
    st = (M * K + gap, K * N + gap, M * N + gap)
    ctx.gemm_batched(a[1], b[1], C[1], T, M, N, K, act=act, strides=st)
    ctx.gemm_batched_bwd(a[1], b[1], y[1], T, M, N, K, act=act, saved=sv[1] if act != "none" else None, dA=dA[1], dB=dB[1], strides=st)
    if act == "none":      # both tiles add in the order of k, as the exact path does
        ex = [up(ctx, np.zeros(x.shape)) for x in (dY, A, B)]
        ctx.gemm_batched(a[1], b[1], ex[0][1], T, M, N, K, strides=st, mode="simt")
        ctx.gemm_batched_bwd(a[1], b[1], y[1], T, M, N, K, dA=ex[1][1], dB=ex[2][1], strides=st, mode="simt")
        for x, e in zip((C, dA, dB), ex):
            assert np.array_equal(ctx.to_numpy(x[0]), ctx.to_numpy(e[0]))
    for t in range(T):
        At, Bt = A[t, :M * K].reshape(M, K), B[t, :K * N].reshape(K, N)
        Yt, St = dY[t, :M * N].reshape(M, N), S[t, :M * N].reshape(M, N)
        dz = oracle.act_bwd(Yt, St, act) if act != "none" else Yt
        z = oracle.gemm(At, Bt, f64=True)
        got = lambda x, n: ctx.to_numpy(x[0]).reshape(T, -1)[t, :n]           # noqa: E731
        check(got(C, M * N).reshape(M, N), oracle.bias_act_fwd(np.asarray(z, np.float32), np.zeros(N, np.float32), act)[0] if act != "none" else z, K, "output")
        check(got(dA, M * K).reshape(M, K), oracle.gemm(dz, Bt, transB=True, f64=True), N, "dA")
        check(got(dB, K * N).reshape(K, N), oracle.gemm(At, dz, transA=True, f64=True), M, "dB")


@pytest.mark.parametrize("M,N,K", [(5, 70, 40), (5, 72, 40), (5, 70, 100)])
def test_infinities_and_nan(ctx, M, N, K):
    # what is outside the tensors does not meet them: an infinity reaches its own row and column, a NaN too, and zeros times them
    A, B = np.ones((M, K), np.float32), np.ones((K, N), np.float32)
    A[1, 3] = np.inf
    A[2, K - 1] = np.nan
    C = ctx.new_tensor((M, N))
    ctx.gemm(up(ctx, A)[1], up(ctx, B)[1], C, M, N, K)
    got = ctx.to_numpy(C)
    assert np.isposinf(got[1]).all() and np.isnan(got[2]).all() and (got[[0, 3, 4]] == K).all()


# Forward products of a short k: where the exact path is the faster one (one k tile of 32 and up to 32 columns, or rows off the 16-byte boundary
# and up to two k tiles) AUTO's sums are in its order, bit for bit; beyond it they are in shares, which an output of thousands of sums shows.
@pytest.mark.parametrize("M,N,K,exact", [(64, 16, 2, True), (1, 1, 1, True), (700, 32, 32, True), (700, 36, 32, False), (700, 33, 64, True), (700, 33, 65, False),
                                         (16384, 17, 8, True), (300, 28, 33, False), (3, 8189, 32, True), (3, 8193, 32, False), (20, 4095, 64, True),
                                         (20, 4097, 64, False), (5000, 17, 40, True), (32768, 32, 3, True)])
@pytest.mark.parametrize("tA,tB", [(False, False), (True, False), (False, True), (True, True)])
def test_forward_of_a_short_k(ctx, oracle, M, N, K, exact, tA, tB):
    r = rng(M + N + K)
    A, B, bias = r.standard_normal((M, K), np.float32), r.standard_normal((K, N), np.float32), r.standard_normal(N, np.float32)
    a, b, v = up(ctx, A.T if tA else A), up(ctx, B.T if tB else B), up(ctx, bias)
    C, P, E = (up(ctx, np.zeros((M, N))) for _ in range(3))
    ctx.gemm(a[1], b[1], C[1], M, N, K, transA=tA, transB=tB, bias=v[1], act="tanh", preact_out=P[1])
    ctx.gemm(a[1], b[1], E[1], M, N, K, transA=tA, transB=tB, bias=v[1], act="none", mode="simt")
    got = ctx.to_numpy(P[0])
    assert np.array_equal(got, ctx.to_numpy(E[0])) == exact
    check(got.reshape(M, N), oracle.gemm(A, B, f64=True).astype(np.float64) + bias, K, "pre-activation")
    check(ctx.to_numpy(C[0]), np.tanh(got.astype(np.float64)), 0, "output")


@pytest.mark.parametrize("T,M,N,K", [(7, 33, 66, 97), (3, 2, 300, 256), (5, 200, 10, 70)])
@pytest.mark.parametrize("gap", [0, 5])
def test_batched_sums_are_in_order_with_an_activation(ctx, T, M, N, K, gap):
    # room between the matrices changes no bit, nor the number of launches: dZ of the whole batch, then the products
    r = rng(T + M)
    f = lambda *s: up(ctx, r.standard_normal(s).astype(np.float32))           # noqa: E731
    st = (M * K + gap, K * N + gap, M * N + gap)
    a, b, y, sv = f(T, st[0]), f(T, st[1]), f(T, st[2]), f(T, st[2])
    out = []
    for mode in ("auto", "simt"):
        dA, dB = up(ctx, np.zeros((T, st[0]))), up(ctx, np.zeros((T, st[1])))
        ctx.gemm_batched_bwd(a[1], b[1], y[1], T, M, N, K, act="gelu", saved=sv[1], dA=dA[1], dB=dB[1], strides=st, mode=mode)
        before = ctx.launch_count()
        ctx.gemm_batched_bwd(a[1], b[1], y[1], T, M, N, K, act="gelu", saved=sv[1], dA=dA[1], dB=dB[1], strides=st, mode=mode)
        assert ctx.launch_count() - before == 3
        out.append((ctx.to_numpy(dA[0]), ctx.to_numpy(dB[0])))
    for x, e in zip(*out):
        assert np.array_equal(x, e)


@pytest.mark.parametrize("M,N,K,act", [(200, 256, 256, "none"), (200, 256, 256, "gelu"), (100, 20, 30, "tanh")])
def test_backward_is_recorded_without_room_for_dz(oracle, M, N, K, act):
    # the gradients take dZ through the activation as they read it: a recording needs no scratch arena of its size
    from ferrograd_b200 import FgError, GpuContext
    c = GpuContext(0)
    c._check(c.lib.fg_ctx_reserve_workspace(c.handle, 1024))
    r = rng(M)
    f = lambda *s: r.standard_normal(s).astype(np.float32)                    # noqa: E731
    A, B, dY, S = f(M, K), f(K, N), f(M, N), np.tanh(f(M, N))
    a, b, y, sv = (up(c, x) for x in (A, B, dY, S))
    dA, dB, db = (up(c, np.zeros(s)) for s in ((M, K), (K, N), (N,)))
    kw = dict(act=act, saved=sv[1] if act != "none" else None)
    c.plan_begin()
    c.gemm_bwd(a[1], b[1], y[1], M, N, K, dA=dA[1], dB=dB[1], dbias=db[1], **kw)
    plan = c.plan_end()
    plan.launch()
    dz = oracle.act_bwd(dY, S, act) if act != "none" else dY
    check(c.to_numpy(dA[0]).reshape(M, K), oracle.gemm(dz, B, transB=True, f64=True), N, "dA")
    check(c.to_numpy(dB[0]).reshape(K, N), oracle.gemm(A, dz, transA=True, f64=True), M, "dB")
    check(c.to_numpy(db[0]), dz.astype(np.float64).sum(0), M, "dbias")
    plan.destroy()
    if N == K and act != "none":      # dA over the saved tensor: dZ is formed first and does need its room
        c.plan_begin()
        with pytest.raises(FgError):
            c.gemm_bwd(a[1], b[1], y[1], M, N, K, dA=sv[1], dB=dB[1], **kw)
        c.plan_end().destroy()
    c.destroy()
