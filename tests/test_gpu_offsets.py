"""Tensors that start off 16-byte boundaries where a kernel reads four words at a time: a bias behind other values in an arena, and results
whose pairs are made by a pass of their own.  Sizes and options send the products through each of the tensor-core kernels."""
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


# split products of f32: 2^-19 of a term from the bf16 rest, and the tensor core's truncating sums of 256 (5e-6 of the result, measured)
TOL = 2e-5


@pytest.mark.parametrize("shift", [1, 2, 3])
@pytest.mark.parametrize("tile", ["auto", "pair", "128x32"])
@pytest.mark.parametrize("M,N,K,mode", [(512, 520, 640, "auto"), (300, 261, 512, "auto"), (2048, 2048, 1024, "auto"), (512, 512, 512, "3xtf32")])
def test_a_bias_off_the_boundary(ctx, oracle, shift, tile, M, N, K, mode):
    r = rng(M + N + K)
    A, B, bias = r.standard_normal((M, K), np.float32), r.standard_normal((K, N), np.float32) * np.float32(K ** -0.5), r.standard_normal(N, np.float32)
    a, b, v, C = up(ctx, A), up(ctx, B), up(ctx, bias, shift), up(ctx, np.zeros((M, N)))
    ctx.set_option("gemm_tile", tile)
    try:
        ctx.gemm(a[1], b[1], C[1], M, N, K, bias=v[1], act="relu", mode=mode)
    finally:
        ctx.set_option("gemm_tile", "auto")
    z = oracle.gemm(A, B, f64=True).astype(np.float64) + bias
    ok, worst = rel_err_ok(ctx.to_numpy(C[0]).reshape(M, N), np.maximum(z, 0), TOL)
    assert ok, f"{worst:.3g}"


@pytest.mark.parametrize("shift", [0, 1, 2])
@pytest.mark.parametrize("M,N,K", [(4096, 10, 512), (300, 101, 1000), (40, 24, 16)])
def test_pairs_of_results_off_the_boundary(ctx, oracle, shift, M, N, K):
    # forward (a narrow layer, a ragged one, a small one) and dA of the layer above, whose pairs are those of what was stored
    from ferrograd_b200.backend import to_bf16_bits
    r = rng(M + N + K)
    A, B, dZ = r.standard_normal((M, K), np.float32), r.standard_normal((K, N), np.float32) * np.float32(K ** -0.5), r.standard_normal((M, N), np.float32)
    a, b, z = up(ctx, A), up(ctx, B), up(ctx, dZ)
    C, dA, dB = up(ctx, np.zeros((M, N)), shift), up(ctx, np.zeros((M, K)), shift), up(ctx, np.zeros((K, N)))
    sc, sa = (M * N + 7) // 8 * 8, (M * K + 7) // 8 * 8
    pc, pa = ctx.new_tensor((2, sc), np.uint16), ctx.new_tensor((2, sa), np.uint16)
    ctx.gemm_paired(a[1], b[1], C[1], M, N, K, C_pairs=pc, C_stride=sc)
    ctx.gemm_bwd_paired(a[1], b[1], z[1], M, N, K, dB=dB[1], dA=dA[1], dA_pairs=pa, dA_stride=sa)
    for x, p, ref, what in ((C, pc, oracle.gemm(A, B, f64=True), "C"), (dA, pa, oracle.gemm(dZ, B, transB=True, f64=True), "dA")):
        got = ctx.to_numpy(x[0])[shift:].reshape(ref.shape)
        ok, worst = rel_err_ok(got, ref, TOL)
        assert ok, f"{what}: {worst:.3g}"
        hi = (got.view(np.uint32) & np.uint32(0xffffe000)).view(np.float32)
        q = ctx.to_numpy(p)[:, :got.size]
        assert np.array_equal(q[0], to_bf16_bits(got).ravel()) and np.array_equal(q[1], to_bf16_bits(got - hi).ravel()), what
