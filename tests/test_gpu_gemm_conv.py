"""The conversion kernel (f32 tensors straight into tensor-core tiles), its K-shares, padded copies and batches: sizes around
tiles of 128 x 64 / 128, k-blocks of 32 and accumulation chunks of 128."""
import numpy as np
import pytest

from conftest import rel_err_ok

pytestmark = pytest.mark.gpu
# Two tensor-core terms per product: the cross terms are rounded to bf16 (2^-18 of the product at most), and up to 64 MMAs
# add into one accumulator with truncation (64 * 2^-24): about 5e-6 of the result's rms, five times that at the worst of
# a million elements.  After an activation, errors of z are compared with the rms of y, which is smaller.
TOL, TOL_ACT = 4e-5, 1e-4


@pytest.fixture(scope="module")
def ctx():
    from ferrograd_b200 import GpuContext
    c = GpuContext(0)
    yield c
    assert c.device_status() == 0
    c.destroy()


def rng(seed):
    return np.random.Generator(np.random.Philox(seed))


def up(ctx, a):
    return ctx.init_tensor_f32(a.shape, np.ascontiguousarray(a, np.float32))


def check(x, ref, tol, what):
    ok, worst = rel_err_ok(x, ref, tol)
    assert ok, f"{what}: {worst:.3g} x {tol}"


# (M, N, K): one tile; edges of tiles; ragged pitches; long K cut into shares; many tiles
SHAPES = [(64, 256, 256), (100, 1000, 1024), (128, 128, 256), (129, 65, 544), (65, 4100, 4096), (200, 333, 77), (257, 130, 8200),
          (1000, 1001, 777), (384, 256, 200), (70, 17, 3600)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("tA,tB", [(False, False), (True, False), (False, True), (True, True)])
def test_forward(ctx, oracle, M, N, K, tA, tB):
    r = rng(M + 3 * N + 7 * K + tA + 2 * tB)
    A, B = r.standard_normal((K, M) if tA else (M, K), np.float32), r.standard_normal((N, K) if tB else (K, N), np.float32) * 0.1
    bias = r.standard_normal(N, np.float32)
    C, P = ctx.new_tensor((M, N)), ctx.new_tensor((M, N))
    ctx.gemm(up(ctx, A), up(ctx, B), C, M, N, K, transA=tA, transB=tB, bias=up(ctx, bias), act="gelu", preact_out=P)
    y, z = oracle.bias_act_fwd(oracle.gemm(A, B, transA=tA, transB=tB, f64=True).astype(np.float32), bias, "gelu")
    check(ctx.to_numpy(P), z, TOL, "pre-activation")
    check(ctx.to_numpy(C), y, TOL_ACT, "output")


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("act,dz_out", [("none", False), ("none", True), ("tanh", False), ("gelu", True)])
def test_backward(ctx, oracle, M, N, K, act, dz_out):
    r = rng(M * 5 + N + K)
    A, B = r.standard_normal((M, K), np.float32), r.standard_normal((K, N), np.float32) * 0.1
    dY, saved = r.standard_normal((M, N), np.float32), np.tanh(r.standard_normal((M, N))).astype(np.float32)
    dz = oracle.act_bwd(dY, saved, act)
    dA, dB, db = ctx.new_tensor((M, K)), ctx.new_tensor((K, N)), ctx.new_tensor((N,))
    Z = ctx.new_tensor((M, N)) if dz_out else None
    Ad, Bd, Yd, Sd = up(ctx, A), up(ctx, B), up(ctx, dY), up(ctx, saved) if act != "none" else None
    ctx.gemm_bwd(Ad, Bd, Yd, M, N, K, act=act, saved=Sd, dA=dA, dB=dB, dbias=db, dZ_out=Z)
    check(ctx.to_numpy(dA), oracle.gemm(dz, B, transB=True, f64=True), TOL, "dA")
    check(ctx.to_numpy(dB), oracle.gemm(A, dz, transA=True, f64=True), TOL, "dB")
    check(ctx.to_numpy(db), dz.astype(np.float64).sum(0), TOL, "dbias")
    if dz_out:
        check(ctx.to_numpy(Z), dz, 1e-5, "dZ")
    only = ctx.new_tensor((K, N))
    ctx.gemm_bwd(Ad, None, Yd, M, N, K, act=act, saved=Sd, dB=only)
    check(ctx.to_numpy(only), oracle.gemm(A, dz, transA=True, f64=True), TOL, "dB alone")


def test_unaligned_operands(ctx, oracle):
    # tensors that start one element off a 16-byte boundary are read from padded copies
    M, N, K = 192, 260, 400
    r = rng(5)
    A, B = r.standard_normal((M, K), np.float32), r.standard_normal((K, N), np.float32) * 0.1
    off = lambda a: up(ctx, np.concatenate([[0], a.ravel()]).astype(np.float32))          # noqa: E731
    Ad, Bd, C = off(A), off(B), ctx.new_tensor((M * N + 1,))
    ctx.gemm(Ad.ptr + 4, Bd.ptr + 4, C.ptr + 4, M, N, K)
    check(ctx.to_numpy(C)[1:].reshape(M, N), oracle.gemm(A, B, f64=True), TOL, "unaligned")


@pytest.mark.parametrize("M,N,K", [(128, 256, 256), (100, 1000, 1024)])
def test_values_that_are_not_finite_stay_in_their_row(ctx, oracle, M, N, K):
    # infinities and NaN make their row of the result not finite and leave the others alone; values whose bf16 plane is finite
    # (below 2^128 - 2^119) are exact to the usual tolerance of their row
    r = rng(M + N)
    A, B = r.standard_normal((M, K), np.float32), r.standard_normal((K, N), np.float32) * 0.1
    A[3, 5], A[40, 0], A[77, K - 1] = np.inf, -np.inf, np.nan
    A[9] = 0.0
    A[9, 2] = np.uint32(0x7f7f7fff).view(np.float32)
    B[2] *= 1e-3
    C = ctx.new_tensor((M, N))
    ctx.gemm(up(ctx, A), up(ctx, B), C, M, N, K)
    got = ctx.to_numpy(C)
    bad = [3, 40, 77]
    assert not np.isfinite(got[bad]).any()
    good = [m for m in range(M) if m not in bad + [9]]
    check(got[good], A[good].astype(np.float64) @ B.astype(np.float64), TOL, "finite rows")
    check(got[9] / 1e30, (A[9, 2].astype(np.float64) / 1e30) * B[2].astype(np.float64), TOL, "row of the largest value")


@pytest.mark.parametrize("T,M,N,K", [(1, 64, 256, 256), (1, 130, 100, 333), (2, 64, 256, 256), (5, 130, 100, 333), (16, 384, 320, 512),
                                     (3, 65, 515, 1024), (40, 64, 64, 1100)])
@pytest.mark.parametrize("gap", [0, 1, 4, 6])
def test_batched(ctx, oracle, T, M, N, K, gap):
    # gap: elements between the matrices of a batch beyond their own size
    r = rng(T + M + N + K + gap)
    act = "tanh" if gap else "none"
    sizes = [M * K + gap, K * N + gap, M * N + gap]
    A, B, dY, S = (r.standard_normal((T, s)).astype(np.float32) for s in (*sizes, sizes[2]))
    B *= 0.1
    S = np.tanh(S)
    a = lambda x, t, shape: x[t, :shape[0] * shape[1]].reshape(shape)                     # noqa: E731
    C, dA, dB = (ctx.init_tensor_f32((T, s), np.full((T, s), 7.0)) for s in (sizes[2], sizes[0], sizes[1]))
    Ad, Bd, Yd, Sd = (up(ctx, x) for x in (A, B, dY, S))
    ctx.gemm_batched(Ad, Bd, C, T, M, N, K, act=act, strides=sizes)
    ctx.gemm_batched_bwd(Ad, Bd, Yd, T, M, N, K, act=act, saved=Sd if act != "none" else None, dA=dA, dB=dB, strides=sizes)
    got, gA, gB = (ctx.to_numpy(x) for x in (C, dA, dB))
    for t in range(T):
        At, Bt = a(A, t, (M, K)), a(B, t, (K, N))
        y, _ = oracle.bias_act_fwd(oracle.gemm(At, Bt, f64=True).astype(np.float32), None, act)
        dz = oracle.act_bwd(a(dY, t, (M, N)), a(S, t, (M, N)), act)
        check(a(got, t, (M, N)), y, TOL_ACT, f"output {t}")
        check(a(gA, t, (M, K)), oracle.gemm(dz, Bt, transB=True, f64=True), TOL, f"dA {t}")
        check(a(gB, t, (K, N)), oracle.gemm(At, dz, transA=True, f64=True), TOL, f"dB {t}")
    if gap:                         # what lies between the matrices is not touched
        assert (got[:, M * N:] == 7.0).all() and (gA[:, M * K:] == 7.0).all() and (gB[:, K * N:] == 7.0).all()


@pytest.mark.parametrize("shift_saved,shift_out", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(128, 512, 512), (100, 256, 1024), (384, 256, 256), (512, 128, 384)])
def test_backward_onto_the_layer_below(ctx, oracle, M, N, K, shift_saved, shift_out):
    # dA * act'(saved) and its column sums in the epilogue, or where a cluster adds its K-shares; the layer below's tensor
    # and dA may start one element off a 16-byte boundary
    r = rng(M + N + K)
    A, B = r.standard_normal((M, K), np.float32), r.standard_normal((K, N), np.float32) * 0.1
    dZ, saved = r.standard_normal((M, N), np.float32), np.tanh(r.standard_normal((M, K))).astype(np.float32)
    place = lambda a, shift: up(ctx, np.concatenate([np.zeros(shift, np.float32), a.ravel()]))          # noqa: E731
    S, dA = place(saved, shift_saved), place(np.zeros((M, K), np.float32), shift_out)
    dB, below = ctx.new_tensor((K, N)), ctx.new_tensor((K,))
    ctx.gemm_bwd_paired(up(ctx, A), up(ctx, B), up(ctx, dZ), M, N, K, dB=dB, dA=dA.ptr + 4 * shift_out, below_act="tanh",
                        below_saved=S.ptr + 4 * shift_saved, below_dbias=below)
    want = oracle.gemm(dZ, B, transB=True, f64=True) * (1.0 - saved.astype(np.float64) ** 2)
    check(ctx.to_numpy(dA)[shift_out:].reshape(M, K), want, TOL, "dA")
    check(ctx.to_numpy(dB), oracle.gemm(A, dZ, transA=True, f64=True), TOL, "dB")
    check(ctx.to_numpy(below), want.sum(0), TOL, "bias gradient of the layer below")


# more samples than outputs and fewer (the longer k is dB's or dA's), more tiles than SMs, both gradients in a launch or one each
@pytest.mark.parametrize("M,N,K", [(1024, 256, 256), (384, 256, 256), (128, 4096, 1024), (2048, 512, 1024), (64, 1024, 1024)])
@pytest.mark.parametrize("how", ["gemm_bwd", "paired", "batched"])
def test_gradient_that_overwrites_the_activation(ctx, oracle, M, N, K, how):
    # dB is complete before dA is written, so dA may be A itself
    T = 4 if how == "batched" else 1
    r = rng(M + N + 3 * K)
    A, B = np.tanh(r.standard_normal((T, M, K))).astype(np.float32), r.standard_normal((T, K, N), np.float32) * 0.1
    dZ = r.standard_normal((T, M, N), np.float32)
    dA = np.stack([oracle.gemm(z, b, transB=True, f64=True) for z, b in zip(dZ, B)])
    dB = np.stack([oracle.gemm(a, z, transA=True, f64=True) for a, z in zip(A, dZ)])
    Bd, Zd = up(ctx, B), up(ctx, dZ)
    for again in range(3):
        x, g = up(ctx, A), ctx.new_tensor((T, K, N))
        if how == "gemm_bwd":
            ctx.gemm_bwd(x, Bd, Zd, M, N, K, dA=x, dB=g)
        elif how == "paired":
            ctx.gemm_bwd_paired(x, Bd, Zd, M, N, K, dB=g, dA=x, below_act="tanh", below_saved=x)
        else:
            ctx.gemm_batched_bwd(x, Bd, Zd, T, M, N, K, dA=x, dB=g)
        check(ctx.to_numpy(g), dB, TOL, "dB")
        check(ctx.to_numpy(x), dA * (1.0 - A.astype(np.float64) ** 2) if how == "paired" else dA, TOL, "dA over A")


# the exact path, a narrow layer, operand planes (one gradient or both), the pair kernel
@pytest.mark.parametrize("M,N,K", [(33, 20, 40), (200, 10, 512), (300, 33, 75), (64, 700, 1021), (2048, 64, 4094), (1024, 1024, 2048)])
@pytest.mark.parametrize("pairs", ["1", "0"])
def test_gradient_that_overwrites_the_saved_tensor(oracle, M, N, K, pairs):
    # dA = (dZ B^T) * act'(saved) may lie over the saved tensor, which is A, on every route
    from ferrograd_b200 import GpuContext
    c = GpuContext(0)
    c.set_option("gemm_pairs", pairs)
    r = rng(M + N + 5 * K)
    A, B = np.tanh(r.standard_normal((M, K))).astype(np.float32), r.standard_normal((K, N), np.float32) * 0.1
    dZ = r.standard_normal((M, N), np.float32)
    x, dB, below = up(c, A), c.new_tensor((K, N)), c.new_tensor((K,))
    c.gemm_bwd_paired(x, up(c, B), up(c, dZ), M, N, K, dB=dB, dA=x, below_act="tanh", below_saved=x, below_dbias=below)
    want = oracle.gemm(dZ, B, transB=True, f64=True) * (1.0 - A.astype(np.float64) ** 2)
    check(c.to_numpy(x), want, TOL, "dA over A")
    check(c.to_numpy(dB), oracle.gemm(A, dZ, transA=True, f64=True), TOL, "dB")
    check(c.to_numpy(below), want.sum(0), TOL, "bias gradient of the layer below")
    assert c.device_status() == 0
    c.destroy()


@pytest.mark.parametrize("T,M,N,K", [(1, 384, 256, 256), (1, 100, 1024, 2048), (9, 384, 512, 320), (1, 1000, 777, 1001)])
def test_products_beside_an_exchange(oracle, T, M, N, K):
    # a communicator of one rank: launches in plain order, units walked by the SMs that the exchange leaves
    import torch  # noqa: F401  (its NCCL is the one that the process loads)
    from ferrograd_b200 import GpuContext
    c = GpuContext(0)
    c.comm_init(1, 0, c.comm_unique_id())
    r = rng(T + M + N + K)
    A, B, dY = (r.standard_normal(s, np.float32) for s in ((T, M, K), (T, K, N), (T, M, N)))
    B *= 0.1
    out, dA, dB, sums = c.new_tensor((T, M, N)), c.new_tensor((T, M, K)), c.new_tensor((T, K, N)), up(c, np.arange(4096.0))
    Ad, Bd, Yd = up(c, A), up(c, B), up(c, dY)
    c.allreduce_sum(sums, 4096)             # in flight until it is joined
    if T > 1:
        c.gemm_batched(Ad, Bd, out, T, M, N, K)
        c.gemm_batched_bwd(Ad, Bd, Yd, T, M, N, K, dA=dA, dB=dB)
    else:
        c.gemm(Ad, Bd, out, M, N, K)
        c.gemm_bwd(Ad, Bd, Yd, M, N, K, dA=dA, dB=dB)
    c.comm_sync(20000)
    got, gA, gB = (c.to_numpy(t) for t in (out, dA, dB))
    for t in range(T):
        check(got[t], oracle.gemm(A[t], B[t], f64=True), TOL, f"output {t}")
        check(gA[t], oracle.gemm(dY[t], B[t], transB=True, f64=True), TOL, f"dA {t}")
        check(gB[t], oracle.gemm(A[t], dY[t], transA=True, f64=True), TOL, f"dB {t}")
    assert (c.to_numpy(sums) == np.arange(4096.0)).all() and c.device_status() == 0
    c.destroy()


@pytest.fixture(params=["64x1", "128x1", "64x2", "128x2", "64x3", "128x3", "64x5", "128x5", "64x8", "128x8"])
def given(request):
    """A context whose f32 products take the conversion kernel with this tile width and these K-shares."""
    from ferrograd_b200 import GpuContext
    c = GpuContext(0)
    c.set_option("gemm_conv", request.param)
    yield c
    assert c.device_status() == 0
    c.destroy()


def n8(n):
    return (n + 7) // 8 * 8


def pairs_of(c, t, n):
    p = c.new_tensor((2, n8(n)), np.uint16)
    c.pairs_from_f32(t, n, p, n8(n))
    return c.to_numpy(p)[:, :n]


# edges of tiles with rows on the 16-byte boundary and off it; more tiles than SMs, with k of their own for either gradient
@pytest.mark.parametrize("M,N,K", [(520, 516, 260), (517, 531, 261), (2100, 540, 1100), (2101, 541, 1101)])
def test_every_tile_and_share(given, oracle, M, N, K):
    c = given
    r = rng(M + N + K)
    A, B = np.tanh(r.standard_normal((M, K))).astype(np.float32), r.standard_normal((K, N), np.float32) * 0.1
    dZ, bias = r.standard_normal((M, N), np.float32), r.standard_normal(N, np.float32)
    Ad, Bd, Zd = up(c, A), up(c, B), up(c, dZ)
    f64 = lambda x: x.astype(np.float64)                                                                # noqa: E731
    # forward: bias, activation, pre-activation, pairs
    C, P, Cp = c.new_tensor((M, N)), c.new_tensor((M, N)), c.new_tensor((2, n8(M * N)), np.uint16)
    c.gemm_paired(Ad, Bd, C, M, N, K, bias=up(c, bias), act="gelu", C_pairs=Cp, C_stride=n8(M * N))
    y, z = oracle.bias_act_fwd((f64(A) @ f64(B)).astype(np.float32), bias, "gelu")
    check(c.to_numpy(C), y, TOL_ACT, "output")
    assert np.array_equal(c.to_numpy(Cp)[:, :M * N], pairs_of(c, C, M * N))
    c.gemm(Ad, Bd, C, M, N, K, bias=up(c, bias), act="gelu", preact_out=P)
    check(c.to_numpy(P), z, TOL, "pre-activation")
    # backward onto the layer below: act' factor, pairs, column sums; both gradients in a launch, then one at a time
    wantA, wantB = (f64(dZ) @ f64(B).T) * (1.0 - f64(A) ** 2), f64(A).T @ f64(dZ)
    dA, dB, below, Ap = c.new_tensor((M, K)), c.new_tensor((K, N)), c.new_tensor((K,)), c.new_tensor((2, n8(M * K)), np.uint16)
    more = dict(below_act="tanh", below_saved=Ad, below_dbias=below, dA_pairs=Ap, dA_stride=n8(M * K))
    before = c.launch_count()
    c.gemm_bwd_paired(Ad, Bd, Zd, M, N, K, dB=dB, dA=dA, **more)
    if N % 4 == 0 and K % 4 == 0:
        assert c.launch_count() - before == 2           # the products, and the fold of the column sums
    gotA, gotB = c.to_numpy(dA), c.to_numpy(dB)
    check(gotA, wantA, TOL, "dA")
    check(gotB, wantB, TOL, "dB")
    check(c.to_numpy(below), wantA.sum(0), TOL, "bias gradient of the layer below")
    assert np.array_equal(c.to_numpy(Ap)[:, :M * K], pairs_of(c, dA, M * K))
    c.gemm_bwd_paired(None, Bd, Zd, M, N, K, dA=dA, **more)
    c.gemm_bwd_paired(Ad, None, Zd, M, N, K, dB=dB)
    assert np.array_equal(c.to_numpy(dA), gotA) and np.array_equal(c.to_numpy(dB), gotB)      # k is long enough for all shares


@pytest.mark.parametrize("T,M,N,K", [(3, 130, 516, 520), (5, 129, 517, 515)])
def test_every_tile_and_share_of_a_batch(given, T, M, N, K):
    r = rng(T + M + N + K)
    A, B, dY = (r.standard_normal(s, np.float32) for s in ((T, M, K), (T, K, N), (T, M, N)))
    Ad, Bd, Yd = up(given, A), up(given, B), up(given, dY)
    C, dA, dB = given.new_tensor((T, M, N)), given.new_tensor((T, M, K)), given.new_tensor((T, K, N))
    given.gemm_batched(Ad, Bd, C, T, M, N, K)
    given.gemm_batched_bwd(Ad, Bd, Yd, T, M, N, K, dA=dA, dB=dB)
    for got, want in ((C, np.matmul(A, B, dtype=np.float64)), (dA, np.matmul(dY, B.transpose(0, 2, 1), dtype=np.float64)),
                      (dB, np.matmul(A.transpose(0, 2, 1), dY, dtype=np.float64))):
        check(given.to_numpy(got), want, TOL, "batch")


def test_batched_refuses_what_one_product_refuses(ctx):
    # an unknown mode and a contraction over nothing: an argument error as from the per-matrix calls, before any launch
    from ferrograd_b200.backend import GEMM_MODE
    M, N, K, T = 256, 256, 256, 4
    t = ctx.new_tensor((T * 256 * 256,))
    p = t.ptr
    before = ctx.launch_count()
    for mode, k in ((7, K), (-1, K), (GEMM_MODE["tf32_bf16x2"], 0)):
        one = ctx.lib.fg_gemm_f32(ctx.handle, mode, 0, 0, M, N, k, p, p, p, None, 0, None)
        assert one != 0
        assert ctx.lib.fg_gemm_batched_f32(ctx.handle, mode, T, M, N, k, p, M * k, p, k * N, p, M * N, None, 0, None) == one
        assert ctx.lib.fg_gemm_batched_bwd_f32(ctx.handle, mode, T, M, N, k, p, M * k, p, k * N, p, M * N, 0, None, p, p) == one
    assert ctx.launch_count() == before


@pytest.mark.parametrize("M,N,K", [(50000, 20, 33), (100000, 32, 64)])
def test_bias_gradient_of_many_samples(ctx, M, N, K):
    # Sums of M values of order one in chains of at most 32 + M / 2048 additions that are added in pairs.  A chain's roundings,
    # 2^-25 of a partial sum that grows with the root of its length, add up to about 2^-25 * sqrt(length / 2) of the chain, and
    # the chains' errors are independent: 2^-25 * sqrt(25) = 1.5e-7 of the 2-norm at the larger size, with half as much again as margin.
    errors = []
    for seed in range(4):
        r = rng(M + seed)
        A, B, dY = r.standard_normal((M, K), np.float32), r.standard_normal((K, N), np.float32), r.standard_normal((M, N), np.float32)
        db, dB = ctx.new_tensor((N,)), ctx.new_tensor((K, N))
        ctx.gemm_bwd(up(ctx, A), up(ctx, B), up(ctx, dY), M, N, K, dB=dB, dbias=db)
        ref = dY.astype(np.float64).sum(0)
        errors.append(np.linalg.norm(ctx.to_numpy(db) - ref) / np.linalg.norm(ref))
    assert np.mean(errors) <= 2.3e-7, errors


@pytest.mark.parametrize("M", [96, 90, 97])
@pytest.mark.parametrize("K", [2044, 2045])
def test_fused_column_sums_in_four_chains(ctx, M, K):
    # Rows on the 16-byte boundary or off it: the same sums, bit for bit.  A block of 32 rows is added in four chains of eight (row
    # r in chain r % 4), which are added in pairs; then the blocks in order.  (N below 64: one k-block or two, no K-shares.)
    N = 24
    r = rng(M + K)
    B, dZ = r.standard_normal((K, N), np.float32), r.standard_normal((M, N), np.float32)
    dA, below = ctx.new_tensor((M, K)), ctx.new_tensor((K,))
    ctx.gemm_bwd_paired(None, up(ctx, B), up(ctx, dZ), M, N, K, dA=dA, below_dbias=below)
    got = ctx.to_numpy(dA)
    want = np.zeros(K, np.float32)
    for m in range(0, M, 32):
        chains = np.zeros((4, K), np.float32)
        for i, row in enumerate(got[m:m + 32]):
            chains[i % 4] += row
        want += (chains[0] + chains[1]) + (chains[2] + chains[3])
    assert np.array_equal(ctx.to_numpy(below), want)


@pytest.mark.parametrize("M,N,K", [(96, 2048, 2048), (128, 1024, 4096), (128, 4096, 1024), (4096, 64, 4096), (16384, 32, 1024), (300, 100, 304)])
@pytest.mark.parametrize("paired", [False, True])
def test_backward_keeps_the_error_of_the_planes(ctx, oracle, M, N, K, paired):
    # Layers of which one gradient does not suit the pair kernel (few samples, few outputs): both gradients keep a rounded
    # main term.  The 2-norm error of a million sums is stable to a percent or so; a truncated main term adds a quarter.
    from ferrograd_b200 import GpuContext
    r = rng(M + N + K)
    A, B = r.standard_normal((M, K), np.float32), r.standard_normal((K, N), np.float32) * 0.1
    dZ = r.standard_normal((M, N), np.float32)
    S = np.tanh(r.standard_normal((M, K))).astype(np.float32)
    z64 = dZ.astype(np.float64)
    refA, refB = z64 @ B.astype(np.float64).T, A.astype(np.float64).T @ z64
    if paired:
        refA *= 1.0 - S.astype(np.float64) ** 2

    def errors(c):
        dA, dB, below = c.new_tensor((M, K)), c.new_tensor((K, N)), c.new_tensor((K,))
        if paired:
            c.gemm_bwd_paired(up(c, A), up(c, B), up(c, dZ), M, N, K, dB=dB, dA=dA, below_act="tanh", below_saved=up(c, S), below_dbias=below)
            check(c.to_numpy(below), refA.sum(0), TOL, "bias gradient of the layer below")
        else:
            c.gemm_bwd(up(c, A), up(c, B), up(c, dZ), M, N, K, dA=dA, dB=dB)
        return [np.linalg.norm(c.to_numpy(g) - ref) / np.linalg.norm(ref) for g, ref in ((dA, refA), (dB, refB))]

    planes = GpuContext(0)
    planes.set_option("gemm_pairs", "0")
    want = errors(planes)
    planes.destroy()
    got = errors(ctx)
    assert got[0] <= 1.08 * want[0] and got[1] <= 1.08 * want[1], (got, want)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("how", ["recording", "out of memory"])
def test_batches_without_scratch_for_all_matrices(oracle, shift, how):
    # dZ of 1001 matrices (66 MB), or padded copies of the operands (330 MB), where the arena cannot grow: they pass through it in
    # parts, it stays where it is, and a plan recorded before can still be launched
    import torch
    from ferrograd_b200 import GpuContext
    T, M, N, K = 1001, 64, 256, 256
    r = rng(T + shift)
    A, B, dY = (r.standard_normal(s, np.float32) for s in ((T, M, K), (T, K, N), (T, M, N)))
    B *= 0.1
    c = GpuContext(0)
    place = lambda a: up(c, np.concatenate([np.zeros(shift, np.float32), a.ravel()]))                   # noqa: E731
    at = lambda t: t.ptr + 4 * shift                                                                    # noqa: E731
    Ad, Bd, Yd = place(A), place(B), place(dY)
    C, dA, dB = place(np.zeros_like(dY)), place(np.zeros_like(A)), place(np.zeros_like(B))

    def both(t):
        c.gemm_batched(at(Ad), at(Bd), at(C), t, M, N, K, act="tanh")
        c.gemm_batched_bwd(at(Ad), at(Bd), at(Yd), t, M, N, K, act="tanh", saved=at(C), dA=at(dA), dB=at(dB))

    def record(t):
        c.plan_begin()
        both(t)
        return c.plan_end()

    c.reserve_workspace(48 << 20)       # what one matrix on the general path takes
    both(40)
    plan = record(40)
    arena = c.workspace_bytes()
    whole = record(T)                   # (and every kernel is loaded before the memory is full)
    whole.launch()
    c.sync()
    whole.destroy()
    if how == "out of memory":
        for t in (C, dA, dB):
            c.memset_zero(t)
        filling, left, size = [], torch.empty(32 << 20, dtype=torch.uint8, device="cuda"), 32 << 30
        try:
            while size >= 16 << 20:
                try:
                    filling.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
                except torch.cuda.OutOfMemoryError:
                    size //= 2
            del left                    # some room is left, too little for the 82 MB that all of dZ would take
            torch.cuda.empty_cache()
            both(T)
            c.sync()
        finally:
            filling.clear()
            torch.cuda.empty_cache()
    assert c.workspace_bytes() == arena < 66 << 20
    got = c.to_numpy(C)[shift:].reshape(T, M, N)
    check(got, np.tanh(np.matmul(A, B, dtype=np.float64)), TOL_ACT, "output")
    dz = dY * (1.0 - got.astype(np.float64) ** 2)
    check(c.to_numpy(dA)[shift:].reshape(T, M, K), np.matmul(dz, B.transpose(0, 2, 1), dtype=np.float64), TOL, "dA")
    check(c.to_numpy(dB)[shift:].reshape(T, K, N), np.matmul(A.transpose(0, 2, 1), dz, dtype=np.float64), TOL, "dB")
    c.memset_zero(C)
    plan.launch()
    check(c.to_numpy(C)[shift:shift + 40 * M * N].reshape(40, M, N), got[:40], TOL, "output of the plan recorded first")
    plan.destroy()
    assert c.device_status() == 0
    c.destroy()
