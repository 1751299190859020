"""Row softmax and the fused loss at the column counts where the kernels change and on rows that start off a 16-byte boundary."""
import numpy as np
import pytest

from conftest import rel_err_ok

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.fixture(scope="module")
def ctx():
    from ferrograd_b200 import GpuContext
    c = GpuContext(0)
    yield c
    c.sync()
    c.destroy()


def check(x, ref, what):
    ok, worst = rel_err_ok(x, ref, TOL)
    assert ok, f"{what}: {worst:.3g}"


@pytest.mark.parametrize("cols", [1, 10, 32, 33, 127, 129, 511, 512, 513, 1001, 4097, 8191, 16383, 16385, 32767, 32769])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows(ctx, oracle, cols, shift):
    rows = 37 if cols < 4097 else 5
    r = np.random.Generator(np.random.Philox(cols + shift))
    x, dy = (2 * r.standard_normal((rows, cols))).astype(np.float32), r.standard_normal((rows, cols)).astype(np.float32)
    base = r.standard_normal((rows, cols)).astype(np.float32)
    labels = r.integers(0, cols + 1, rows).astype(np.uint32)          # a label of `cols` is out of range: no loss, no one-hot
    n = rows * cols

    def place(a):
        return ctx.init_tensor_f32((n + shift,), np.concatenate([np.zeros(shift, np.float32), a.ravel()]))

    at = lambda t: t.ptr + 4 * shift                                           # noqa: E731
    take = lambda t: ctx.to_numpy(t)[shift:].reshape(rows, cols)               # noqa: E731
    xd, dyd, y = place(x), place(dy), place(np.zeros(n, np.float32))
    ctx.softmax_fwd(at(xd), at(y), rows, cols)
    yref = oracle.softmax_fwd(x)
    check(take(y), yref, "softmax")
    for accumulate in (False, True):
        dx = place(base)
        ctx.softmax_bwd(at(y), at(dyd), at(dx), rows, cols, accumulate=accumulate)
        ref = oracle.softmax_bwd(yref, dy)
        check(take(dx), base + ref if accumulate else ref, f"softmax backward, accumulate {accumulate}")
    loss, mean, dl, probs = ctx.new_tensor((rows,)), ctx.new_tensor((1,)), place(np.zeros(n, np.float32)), place(np.zeros(n, np.float32))
    am, lab = ctx.new_tensor((rows,), np.uint32), ctx.init_tensor_u32((rows,), labels)
    ctx.softmax_ce(at(xd), lab, rows, cols, grad_scale=0.5, loss_row=loss, loss_mean=mean, dlogits=at(dl), probs=at(probs), argmax=am)
    x64 = x.astype(np.float64)
    logp = x64 - x64.max(1, keepdims=True)
    logp -= np.log(np.exp(logp).sum(1, keepdims=True))
    inside = labels < cols
    onehot = np.zeros((rows, cols))
    onehot[np.arange(rows)[inside], labels[inside]] = 1.0
    want = np.where(inside, -logp[np.arange(rows), np.minimum(labels, cols - 1)], 0.0)
    check(ctx.to_numpy(loss), want, "loss")
    check(take(probs), np.exp(logp), "probabilities")
    check(take(dl), (np.exp(logp) - onehot) * 0.5, "gradient")
    assert np.array_equal(ctx.to_numpy(am), x.argmax(1))


@pytest.mark.parametrize("cols", [100, 512, 600, 2049, 4096, 8193, 16385])
@pytest.mark.parametrize("rows", [21, 300])
def test_tensors_that_lie_differently(ctx, oracle, rows, cols):
    # each tensor off a 16-byte boundary by another number of elements: the kernels that stream a row, by words
    r = np.random.Generator(np.random.Philox(cols))
    x, dy, base = ((2 * r.standard_normal((rows, cols))).astype(np.float32) for _ in range(3))
    labels = r.integers(0, cols, rows).astype(np.uint32)

    def place(a, shift):
        t = ctx.init_tensor_f32((a.size + shift,), np.concatenate([np.full(shift, 7.0, np.float32), a.ravel()]))
        return t, t.ptr + 4 * shift, lambda: ctx.to_numpy(t)[shift:].reshape(rows, cols)

    (_x, xp, _), (_d, dp, _), (_y, yp, y), (_g, gp, g) = place(x, 0), place(dy, 1), place(base, 2), place(base, 3)
    ctx.softmax_fwd(xp, yp, rows, cols)
    yref = oracle.softmax_fwd(x)
    check(y(), yref, "softmax")
    ctx.softmax_bwd(yp, dp, gp, rows, cols)
    check(g(), oracle.softmax_bwd(yref, dy), "softmax backward")
    ctx.softmax_bwd(yp, dp, gp, rows, cols, accumulate=True)
    check(g(), 2 * oracle.softmax_bwd(yref, dy), "softmax backward, accumulated")
    (_p, pp, probs), (_l, lp, dl) = place(base, 1), place(base, 2)
    loss, mean, am = ctx.new_tensor((rows,)), ctx.new_tensor((1,)), ctx.new_tensor((rows,), np.uint32)
    ctx.softmax_ce(xp, ctx.init_tensor_u32((rows,), labels), rows, cols, grad_scale=0.5, loss_row=loss, loss_mean=mean, dlogits=lp,
                   probs=pp, argmax=am)
    onehot = np.zeros((rows, cols), np.float32)
    onehot[np.arange(rows), labels] = 1.0
    check(probs(), yref, "probabilities")
    check(dl(), (yref - onehot) * np.float32(0.5), "gradient")
    assert np.array_equal(ctx.to_numpy(am), x.argmax(1))


@pytest.mark.parametrize("cols", [20, 300, 1003])
def test_masked_columns_and_in_place(ctx, cols):
    # -inf logits (a mask) get probability zero; the type's lowest value does too; y may be x
    rows = 9
    r = np.random.Generator(np.random.Philox(cols))
    x = r.standard_normal((rows, cols)).astype(np.float32)
    x[:, ::3] = -np.inf
    x[:, 1::3] = np.finfo(np.float32).min
    t = ctx.init_tensor_f32((rows, cols), x)
    ctx.softmax_fwd(t, t, rows, cols)
    x64 = x.astype(np.float64)
    e = np.exp(x64 - x64.max(1, keepdims=True))
    check(ctx.to_numpy(t), e / e.sum(1, keepdims=True), "masked softmax")


# The mean of the losses is added by the last of up to two blocks per SM (of eight rows, or of one), or by a launch of its own.
@pytest.mark.parametrize("rows,cols", [(1, 10), (295, 30), (2368, 129), (2369, 511), (295, 512), (297, 4096), (296, 1001), (300, 5001), (2, 8192), (700, 32768),
                                       (40, 32769)])
def test_mean_of_the_losses(ctx, rows, cols):
    r = np.random.Generator(np.random.Philox(rows * cols))
    x, lab = ctx.init_tensor_f32((rows, cols), r.standard_normal((rows, cols)).astype(np.float32)), r.integers(0, cols, rows).astype(np.uint32)
    loss, mean, labels = ctx.new_tensor((rows,)), ctx.new_tensor((1,)), ctx.init_tensor_u32((rows,), lab)
    for _ in range(2):
        ctx.softmax_ce(x, labels, rows, cols, loss_row=loss, loss_mean=mean)
        # positive terms, added in chains of rows / 32 at most and trees: (rows / 32 + 16) roundings at most
        want = ctx.to_numpy(loss).astype(np.float64).mean()
        assert abs(float(ctx.to_numpy(mean)[0]) - want) <= 2.0 ** -24 * (rows / 32 + 16) * want
