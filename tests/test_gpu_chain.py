"""Elementwise programs as the chain kernel runs them: random programs, lengths around the groups of four and the blocks of
1024, unaligned tensors, several loads of one input, unused inputs, accumulation."""
import numpy as np
import pytest

from conftest import rel_err_ok

pytestmark = pytest.mark.gpu

BINARY, UNARY = ("add", "sub", "mul", "div"), ("neg", "abs", "tanh", "relu", "gelu", "elu", "exp", "log")


@pytest.fixture(scope="module")
def ctx():
    from ferrograd_b200 import GpuContext
    c = GpuContext(0)
    yield c
    c.sync()
    c.destroy()


def random_program(r, length, ninputs):
    """Values stay away from zero denominators and overflow: div and log read an input (positive), exp reads a tanh."""
    prog, inputs, tanhs = [("input", 0, 0, 0.0)], [0], []
    while len(prog) < length:
        k, kind = len(prog), r.integers(0, 8)
        if kind == 0 and k < length - 1:
            prog.append(("input", int(r.integers(0, ninputs)), 0, 0.0))
            inputs.append(k)
        elif kind == 1 and k < length - 1:
            prog.append(("const", 0, 0, float(np.float32(r.uniform(-1, 1)))))
        elif kind <= 4:
            op = BINARY[r.integers(0, 4)]
            b = int(r.choice(inputs)) if op == "div" else int(r.integers(0, k))
            if op == "mul":             # products of products would grow without bound
                b = int(r.choice(inputs))
            prog.append((op, k - 1 if r.integers(0, 2) else int(r.integers(0, k)), b, 0.0))
        else:
            op = UNARY[r.integers(0, 8)]
            a = int(r.integers(0, k))
            if op == "log":
                a = int(r.choice(inputs))
            if op == "exp":
                if not tanhs:
                    op = "tanh"
                else:
                    a = int(r.choice(tanhs))
            if op == "tanh":
                tanhs.append(k)
            prog.append((op, a, 0, 0.0))
    return prog


@pytest.mark.parametrize("n", [1, 3, 4, 515, 1023, 1028, 2051, 70001])
@pytest.mark.parametrize("shift", [0, 1])
def test_random_programs(ctx, oracle, n, shift):
    r = np.random.Generator(np.random.Philox(n * 2 + shift))
    for length in (1, 2, 5, 12, 24):
        ninputs = int(r.integers(1, 5))
        prog = random_program(r, length, ninputs)
        x = [(np.abs(r.standard_normal(n)) * 0.5 + 0.75).astype(np.float32) for _ in range(ninputs)]
        seed = r.standard_normal(n).astype(np.float32)

        def place(a):       # shift = 1: one element past a 16-byte boundary
            return ctx.init_tensor_f32((n + shift,), np.concatenate([np.zeros(shift, np.float32), a]))

        at = lambda t: t.ptr + 4 * shift                                   # noqa: E731
        take = lambda t: ctx.to_numpy(t)[shift:]                           # noqa: E731
        xd, sd, out = [place(a) for a in x], place(seed), place(np.zeros(n, np.float32))
        k = int(r.integers(0, length))
        kept = place(np.zeros(n, np.float32))
        ctx.eltwise_chain_fwd(prog, [at(t) for t in xd], at(out), n, saved={k: at(kept)})
        ref, saved = oracle.eltwise_fwd(prog, x, save=(k,))
        # each of up to 24 operations contributes a few units of 2^-24 of values of order one
        for got, want in ((take(out), ref), (take(kept), saved[k])):
            ok, worst = rel_err_ok(got, want, 2e-5)
            assert ok, (prog, worst)
        base = [r.standard_normal(n).astype(np.float32) for _ in range(ninputs)]
        gref = oracle.eltwise_bwd(prog, x, seed)
        for accumulate in (False, True):
            gd = [place(b) for b in base]
            want_grad = [bool(r.integers(0, 4)) for _ in range(ninputs)]
            ctx.eltwise_chain_bwd(prog, [at(t) for t in xd], at(sd), [at(g) if w else None for g, w in zip(gd, want_grad)], n,
                                  accumulate=accumulate)
            for g, w, b, gr in zip(gd, want_grad, base, gref):
                ok, worst = rel_err_ok(take(g), (b + gr if accumulate else gr) if w else b, 5e-5)
                assert ok, (prog, accumulate, worst)


def test_output_may_overwrite_an_input(ctx, oracle):
    r = np.random.Generator(np.random.Philox(9))
    n = 5003
    w, g = r.standard_normal(n).astype(np.float32), r.standard_normal(n).astype(np.float32)
    prog = [("input", 0, 0, 0.0), ("input", 1, 0, 0.0), ("const", 0, 0, 0.5), ("mul", 1, 2, 0.0), ("sub", 0, 3, 0.0)]
    wd = ctx.init_tensor_f32((n,), w)
    ctx.eltwise_chain_fwd(prog, [wd, ctx.init_tensor_f32((n,), g)], wd, n)
    assert np.array_equal(ctx.to_numpy(wd), oracle.eltwise_fwd(prog, [w, g])[0])


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
def test_gelu_of_extreme_values(ctx, dtype):
    # the limits: x for large positive, zero for large negative, NaN stays NaN, +inf stays +inf; its derivative 1, 0 and 1/2 at zero
    small = 1e-3 if dtype == "f16" else 1e-6            # a normal number of the type
    x = np.array([0.0, -0.0, 30.0, -30.0, 3e4, -3e4, np.inf, np.nan, small, -small], np.float32)
    n = x.size
    init = {"f32": ctx.init_tensor_f32, "f16": ctx.init_tensor_f16, "bf16": ctx.init_tensor_bf16}[dtype]
    prog = [("input", 0, 0, 0.0), ("gelu", 0, 0, 0.0)]
    t, out, grad, ones = init((n,), x), init((n,), np.zeros(n)), init((n,), np.zeros(n)), init((n,), np.ones(n))
    ctx.eltwise_chain_fwd(prog, [t], out, n, dtype=dtype)
    ctx.eltwise_chain_bwd(prog, [t], ones, [grad], n, dtype=dtype)

    def down(v):
        back = ctx.new_tensor((n,))
        ctx.convert(v, dtype, back, "f32", n)
        return ctx.to_numpy(back)

    y, x, g = down(out), down(t), down(grad)
    # gelu(x) / x = 1/2 + 0.4 x near zero; one rounding of the type (2^-9 in bf16) for x and one for the result
    near = {"f32": 1e-5, "f16": 2e-3, "bf16": 8e-3}[dtype]
    assert y[0] == 0 and y[1] == 0 and y[2] == x[2] and y[3] == 0 and y[4] == x[4] and y[5] == 0 and np.isposinf(y[6]) and np.isnan(y[7])
    assert np.allclose(y[8:], 0.5 * x[8:], rtol=near, atol=0)
    assert g[0] == 0.5 and g[1] == 0.5 and g[2] == 1 and g[3] == 0 and g[4] == 1 and g[5] == 0 and np.isnan(g[7])
    assert np.allclose(g[8:], 0.5, rtol=near, atol=0)
    if dtype == "f32":                                  # the activation's backward pass on its own
        dz = ctx.new_tensor((n,))
        ctx.act_bwd(ones, t, dz, n, "gelu")
        assert np.array_equal(ctx.to_numpy(dz), g, equal_nan=True)


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("n", [7, 2048, 2049, 4097, 50003])
@pytest.mark.parametrize("shift", [0, 1])
def test_packed_arithmetic_rounds_as_single_steps_do(ctx, dtype, n, shift):
    # + - * / on 16-bit elements, two at a time or not, equals the f32 operation followed by one rounding: bit for bit, with
    # subnormals, infinities and NaN among the values; tiles of 2048, an incomplete last one, tensors off the boundary of four
    import torch
    td = {"f16": torch.float16, "bf16": torch.bfloat16}[dtype]
    gen = torch.Generator().manual_seed(n + shift)
    special = torch.tensor([0.0, -0.0, float("inf"), float("-inf"), float("nan"), 1e-7, -1e-7, 6e4, -6e4, 1e-39, -1e-39, 1.0])

    def values():
        v = torch.randn(n, generator=gen)
        at = torch.randint(0, n, (max(1, n // 5),), generator=gen)
        v[at] = special[torch.randint(0, len(special), (len(at),), generator=gen)]
        return v.to(td)

    x, y, g = values(), values(), values()
    place = lambda v: torch.cat([torch.zeros(shift, dtype=td), v]).cuda()   # noqa: E731
    r = lambda v: v.to(td).float()                                          # noqa: E731
    xf, yf, gf = x.float(), y.float(), g.float()
    prog = [("input", 0, 0, 0.0), ("input", 1, 0, 0.0), ("add", 0, 1, 0.0), ("mul", 2, 0, 0.0), ("sub", 1, 3, 0.0), ("div", 4, 1, 0.0),
            ("neg", 5, 0, 0.0), ("abs", 4, 0, 0.0), ("add", 6, 7, 0.0), ("relu", 8, 0, 0.0)]
    a = r(xf + yf)
    m = r(a * xf)
    d = r(yf - m)
    t = r(-r(d / yf) + d.abs())
    want = torch.where(t > 0, t, torch.zeros_like(t)).to(td)
    xd, yd, gd, out, dx, dy = (place(v) for v in (x, y, g, torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(x)))
    torch.cuda.synchronize()
    p = lambda v: v.data_ptr() + 2 * shift                                  # noqa: E731
    ctx.eltwise_chain_fwd(prog, [p(xd), p(yd)], p(out), n, dtype=dtype)
    ctx.sync()
    same = lambda u, v: torch.equal(torch.nan_to_num(u, nan=123.0), torch.nan_to_num(v, nan=123.0)) and torch.equal(u.isnan(), v.isnan())  # noqa: E731
    assert same(out.cpu()[shift:], want)
    ctx.eltwise_chain_bwd([("input", 0, 0, 0.0), ("input", 1, 0, 0.0), ("mul", 0, 1, 0.0), ("relu", 2, 0, 0.0)], [p(xd), p(yd)], p(gd),
                          [p(dx), p(dy)], n, dtype=dtype)
    ctx.sync()
    adj = gf * (r(xf * yf) > 0).float()
    assert same(dx.cpu()[shift:], (adj * yf).to(td)) and same(dy.cpu()[shift:], (adj * xf).to(td))


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("per_sm,per_block", [(2, 4), (5, 4)])
def test_threads_with_four_words_and_with_eight_do_the_same(ctx, dtype, shift, per_sm, per_block):
    # one element below, at and above the size up to which a thread has four words (two or five blocks per SM): the same elements
    # have the same results, forward and backward, whatever the split
    import torch
    td = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[dtype]
    edge = torch.cuda.get_device_properties(0).multi_processor_count * per_sm * 128 * per_block * (1 if dtype == "f32" else 2)
    prog = [("input", 0, 0, 0.0), ("input", 1, 0, 0.0), ("add", 0, 1, 0.0)]
    if per_sm == 5:
        prog = prog[:2] + [("exp", 0, 0, 0.0), ("const", 0, 0, 1.5), ("add", 2, 3, 0.0), ("div", 1, 4, 0.0), ("gelu", 5, 0, 0.0), ("mul", 6, 0, 0.0)]
    gen = torch.Generator().manual_seed(edge + shift)
    place = lambda v: torch.cat([torch.zeros(shift, dtype=td), v.to(td)]).cuda()          # noqa: E731
    x, y, g = (place(torch.randn(edge + 1, generator=gen)) for _ in range(3))
    p = lambda v: v.data_ptr() + shift * v.element_size()                                 # noqa: E731
    seen = []
    for n in (edge - 1, edge, edge + 1):
        out, dx, dy = (torch.full((edge + 1 + shift,), 7.0, dtype=td, device="cuda") for _ in range(3))
        torch.cuda.synchronize()
        ctx.eltwise_chain_fwd(prog, [p(x), p(y)], p(out), n, dtype=dtype)
        ctx.eltwise_chain_bwd(prog, [p(x), p(y)], p(g), [p(dx), p(dy)], n, dtype=dtype)
        ctx.sync()
        for v in (out, dx, dy):
            assert (v[shift + n:] == 7.0).all() and (v[:shift] == 7.0).all()
        seen.append([v[shift:shift + edge - 1].clone() for v in (out, dx, dy)])
    assert all(torch.equal(a, b) for a, b in zip(seen[0], seen[1])) and all(torch.equal(a, b) for a, b in zip(seen[0], seen[2]))
    if per_sm == 2:
        assert torch.equal(seen[0][0], (x + y)[shift:shift + edge - 1])
