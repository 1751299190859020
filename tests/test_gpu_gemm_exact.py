"""The exact path at the edges of its two tiles (64 x 64, 16 x 32) and k tiles (32)."""
import numpy as np
import pytest

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


def up(ctx, a):
    return ctx.init_tensor_f32(a.shape, np.ascontiguousarray(a, np.float32))


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (1, 1000, 700), (15, 33, 31), (16, 32, 32), (17, 31, 65), (63, 515, 300), (640, 1300, 40)])
@pytest.mark.parametrize("tA,tB", [(False, False), (True, False), (False, True), (True, True)])
def test_exact_path(ctx, oracle, M, N, K, tA, tB):
    # both tiles of the exact path: bit for bit the sequential fma chain
    r = rng(M + N + K)
    A, B = r.standard_normal((K, M) if tA else (M, K), np.float32), r.standard_normal((N, K) if tB else (K, N), np.float32)
    bias = r.standard_normal(N, np.float32)
    C, P = ctx.new_tensor((M, N)), ctx.new_tensor((M, N))
    ctx.gemm(up(ctx, A), up(ctx, B), C, M, N, K, transA=tA, transB=tB, bias=up(ctx, bias), act="relu", preact_out=P, mode="simt")
    y, z = oracle.bias_act_fwd(oracle.gemm(A, B, transA=tA, transB=tB), bias, "relu")
    assert np.array_equal(ctx.to_numpy(P), z) and np.array_equal(ctx.to_numpy(C), y)
