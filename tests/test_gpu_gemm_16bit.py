"""16-bit products read as they lie (K-major or MN-major) or from padded copies: sizes around tiles of 256, k-blocks of 64 and
pitches that are no multiple of 16 bytes."""
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


def check(x, ref, tol, what):
    ok, worst = rel_err_ok(x, ref, tol)
    assert ok, f"{what}: {worst:.3g} x {tol}"


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("M,N,K", [(64, 64, 64), (256, 512, 192), (130, 264, 1100), (257, 100, 72), (63, 1001, 515), (512, 8, 2048)])
@pytest.mark.parametrize("act", ["none", "gelu"])
def test_16bit_as_it_lies(ctx, oracle, dtype, M, N, K, act):
    r = rng(M + N * 3 + K * 5)
    rd = lambda a: oracle.round_to(a.astype(np.float32), dtype)                           # noqa: E731
    init = ctx.init_tensor_f16 if dtype == "f16" else ctx.init_tensor_bf16
    A, B, dY, S = rd(r.standard_normal((M, K))), rd(r.standard_normal((K, N)) * 0.1), rd(r.standard_normal((M, N))), rd(r.standard_normal((M, N)))
    t16 = lambda shape: ctx.new_tensor(shape, np.float16 if dtype == "f16" else np.uint16)       # noqa: E731

    def down(t):
        out = ctx.new_tensor(t.shape)
        ctx.convert(t, dtype, out, "f32", t.size)
        return ctx.to_numpy(out)

    C, dA, dB, db = t16((M, N)), t16((M, K)), t16((K, N)), t16((N,))
    Ad, Bd, Yd, Sd = (init(x.shape, x) for x in (A, B, dY, S))
    ctx.gemm_lowp(Ad, Bd, C, M, N, K, dtype, act="none")
    tol = 2.0 ** -10 if dtype == "f16" else 2.0 ** -7            # one unit of the storage type
    check(down(C), oracle.gemm(A, B, f64=True), tol, "output")
    ctx.gemm_bwd_lowp(Ad, Bd, Yd, M, N, K, dtype, act=act, saved=Sd if act != "none" else None, dA=dA, dB=dB, dbias=db)
    dz = rd(oracle.act_bwd(dY, S, act))
    check(down(dA), oracle.gemm(dz, B, transB=True, f64=True), 2 * tol, "dA")
    check(down(dB), oracle.gemm(A, dz, transA=True, f64=True), 2 * tol, "dB")
    check(down(db), dz.astype(np.float64).sum(0), 2 * tol, "dbias")
