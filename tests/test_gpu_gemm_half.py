"""Sixteen-bit products in 128 x 128 and 128 x 64 tiles with K-shares: sizes around the tiles, k-blocks of 64, chunks of 1024 and shares,
one product and both gradients in a launch, outputs whose rows start on eight bytes and off them."""
import numpy as np
import pytest

from conftest import rel_err_ok

pytestmark = pytest.mark.gpu
PLANS = ["auto", "64x1", "128x1", "64x2", "128x3", "64x8", "128x8"]


@pytest.fixture(scope="module")
def ctx():
    from ferrograd_b200 import GpuContext
    c = GpuContext(0)
    yield c
    assert c.device_status() == 0
    c.destroy()


@pytest.fixture(params=PLANS)
def plan(ctx, request):
    ctx.set_option("gemm_conv", request.param)
    yield request.param
    ctx.set_option("gemm_conv", "auto")


def rng(seed):
    return np.random.Generator(np.random.Philox(seed))


def check(x, ref, tol, what):
    ok, worst = rel_err_ok(x, ref, tol)
    assert ok, f"{what}: {worst:.3g} x {tol}"


class Half:
    """Tensors of one storage type."""

    def __init__(self, ctx, oracle, dtype):
        self.ctx, self.dtype = ctx, dtype
        self.round = lambda a: oracle.round_to(np.asarray(a, np.float32), dtype)
        self.unit = 2.0 ** -10 if dtype == "f16" else 2.0 ** -7

    def up(self, a):
        return (self.ctx.init_tensor_f16 if self.dtype == "f16" else self.ctx.init_tensor_bf16)(a.shape, a)

    def new(self, *shape):
        return self.ctx.new_tensor(shape, np.float16 if self.dtype == "f16" else np.uint16)

    def down(self, t):
        out = self.ctx.new_tensor(t.shape)
        self.ctx.convert(t, self.dtype, out, "f32", t.size)
        return self.ctx.to_numpy(out)


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (64, 64, 64), (128, 128, 128), (129, 65, 200), (98, 384, 471), (300, 100, 1100), (257, 130, 2112), (40, 1001, 64),
                                   (2100, 72, 40)])
def test_forward(ctx, oracle, plan, dtype, M, N, K):
    h, r = Half(ctx, oracle, dtype), rng(M + N * 3 + K * 5)
    A, B, bias = h.round(r.standard_normal((M, K))), h.round(r.standard_normal((K, N)) * K ** -0.5), h.round(r.standard_normal(N))
    C, P = h.new(M, N), h.new(M, N)
    ctx.gemm_lowp(h.up(A), h.up(B), C, M, N, K, dtype, bias=h.up(bias), act="gelu", preact_out=P)
    z = oracle.gemm(A, B, f64=True).astype(np.float64) + bias
    y, _ = oracle.bias_act_fwd(np.asarray(z, np.float32), np.zeros(N, np.float32), "gelu")
    check(h.down(P), z, h.unit, "pre-activation")       # one rounding to storage
    check(h.down(C), y, h.unit, "output")


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("M,N,K", [(64, 64, 64), (130, 264, 100), (504, 316, 1264), (196, 992, 1216), (98, 384, 471), (1100, 72, 136), (85, 1031, 336)])
@pytest.mark.parametrize("act", ["none", "tanh"])
def test_backward(ctx, oracle, plan, dtype, M, N, K, act):
    h, r = Half(ctx, oracle, dtype), rng(M + N * 3 + K * 5)
    A, B, dY, S = h.round(r.standard_normal((M, K))), h.round(r.standard_normal((K, N)) * 0.1), h.round(r.standard_normal((M, N))), h.round(np.tanh(r.standard_normal((M, N))))
    a, b, y, s = h.up(A), h.up(B), h.up(dY), h.up(S) if act != "none" else None
    dz = h.round(oracle.act_bwd(dY, S, act)) if act != "none" else dY
    refs = oracle.gemm(dz, B, transB=True, f64=True), oracle.gemm(A, dz, transA=True, f64=True), dz.astype(np.float64).sum(0)

    def same(dA, dB, db, what):
        for t, ref, name in zip((dA, dB, db), refs, ("dA", "dB", "dbias")):
            if t is not None:
                check(h.down(t), ref, h.unit, what + name)

    dA, dB, db = h.new(M, K), h.new(K, N), h.new(N)
    ctx.gemm_bwd_lowp(a, b, y, M, N, K, dtype, act=act, saved=s, dA=dA, dB=dB, dbias=db)
    same(dA, dB, db, "")
    both = h.down(dA), h.down(dB)
    dA, dB = h.new(M, K), h.new(K, N)
    ctx.gemm_bwd_lowp(a, None, y, M, N, K, dtype, act=act, saved=s, dB=dB)
    ctx.gemm_bwd_lowp(None, b, y, M, N, K, dtype, act=act, saved=s, dA=dA)
    same(dA, dB, None, "one by one, ")
    if plan in ("64x1", "128x1"):      # k whole, together and apart (shares shrink with the shorter k of the two)
        assert np.array_equal(h.down(dA), both[0]) and np.array_equal(h.down(dB), both[1])
    # the gradient of A over A: dB is complete before
    dB = h.new(K, N)
    ctx.gemm_bwd_lowp(a, b, y, M, N, K, dtype, act=act, saved=s, dA=a, dB=dB, dbias=db)
    same(a, dB, db, "over A, ")


def test_the_pair_kernel_reads_a_16bit_bias(ctx, oracle):
    # tiles of 256 x 256, with K-shares folded by a launch of their own (k of 4096 on few tiles) and without
    ctx.set_option("gemm_tile", "pair")
    for dtype in ("bf16", "f16"):
        for M, N, K in ((256, 520, 64), (300, 261, 4096)):
            h, r = Half(ctx, oracle, dtype), rng(N)
            A, B, bias = h.round(r.standard_normal((M, K))), h.round(r.standard_normal((K, N)) * K ** -0.5), h.round(r.standard_normal(N))
            C = h.new(M, N)
            ctx.gemm_lowp(h.up(A), h.up(B), C, M, N, K, dtype, bias=h.up(bias))
            check(h.down(C), oracle.gemm(A, B, f64=True).astype(np.float64) + bias, h.unit, "output")
    ctx.set_option("gemm_tile", "auto")
