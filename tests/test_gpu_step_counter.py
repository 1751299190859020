"""AdamW's step counter, which the update of a dispatch moves itself: one launch's tensors (16), one more, and three launches of them."""
import numpy as np
import pytest

from conftest import rel_err_ok

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tensors", [1, 16, 17, 33])
@pytest.mark.parametrize("plans", ["0", "1"])
def test_every_dispatch_is_one_step(oracle, tensors, plans):
    from ferrograd_b200 import MEAN_SQUARED_ERROR, GpuContext, Graph, Metadata, Optim, f32_bits
    ctx = GpuContext(0)
    ctx.set_option("exec_plans", plans)
    n, lr, opt = 8, 1e-2, Optim.adamw()
    shape = (n, n)
    r = np.random.Generator(np.random.Philox(tensors))
    meta = Metadata.new()
    field = meta.new_field()
    graph = Graph.new(MEAN_SQUARED_ERROR, opt.lower)
    g = graph.define_ops()
    y, *factors = [g.input([field, field]) for _ in range(tensors + 1)]      # (nodes 0, 1, ...)
    for f in factors:
        y = g.matmul(y, f)
    saved = graph.compute_saved_nodes()
    graph.validate(meta)
    binding = [f32_bits(lr), n]
    t = ctx.alloc_tensors(graph, saved, ctx.alloc_meta(binding), opt.state)
    kernels = ctx.compile(graph.lower(meta, None, saved), None)
    w = [(np.eye(n) + 0.1 * r.standard_normal(shape)).astype(np.float32) for _ in range(tensors + 1)]
    ins = [ctx.init_tensor_f32(shape, a) for a in w]
    sch = ctx.schedule(kernels, binding, ins, t, [], opt.state, trainable=[0] + [1] * tensors)
    target = ctx.init_tensor_f32(shape, r.standard_normal(shape).astype(np.float32))
    m, v = [np.zeros(shape, np.float32) for _ in w], [np.zeros(shape, np.float32) for _ in w]
    for step in (1, 2, 3, 4):
        ctx.dispatch_forward(sch)
        ctx.dispatch_loss(sch, target)
        ctx.dispatch_backward(sch)
        grads = {node: ctx.download(t.grad_tensors[i], np.empty(shape, np.float32)) for i, node in enumerate(t.grad_nodes)}
        before = [ctx.to_numpy(x).copy() for x in ins]
        ctx.dispatch_optim(sch)
        for k in range(1, tensors + 1):
            ref = before[k]
            oracle.adamw(ref, np.ascontiguousarray(grads[k]), m[k], v[k], lr, *opt.state, step)
            # a step of about lr whose correction, 1 - beta2^step, is off by half for a step counted wrongly; in f32 powf(beta2) and the
            # subtraction from one lose 2^-24 / 1e-3 of it, and the root halves that: 3e-5 of a step of 1e-2 on weights of rms 0.4: 1e-6
            ok, worst = rel_err_ok(ctx.to_numpy(ins[k]), ref, 1e-6)
            assert ok, f"tensor {k} after step {step}: {worst:.3g}"
    t.destroy()
    ctx.destroy()


# A beta outside [0, 1) has no bias correction: the update is refused, before a weight, a moment or the counter changes, by plain launches
# and by recorded ones (whose first dispatch is eager).  With the betas mended the same gradients make step one.
@pytest.mark.parametrize("beta1,beta2", [(1.0, 0.999), (0.9, 1.0), (-0.1, 0.999), (0.9, float("nan"))])
@pytest.mark.parametrize("plans", ["0", "1"])
def test_betas_out_of_range_are_refused(oracle, beta1, beta2, plans):
    import ctypes as C

    from ferrograd_b200 import FgError, GpuContext, _lib
    from ferrograd_b200.mlp import GraphMLP
    ctx = GpuContext(0)
    ctx.set_option("exec_plans", plans)
    dims, batch, lr = [4, 8, 2], 16, 1e-2
    r = np.random.Generator(np.random.Philox(3))
    net = GraphMLP(ctx, dims, batch, "tanh", "mse", ("adamw", lr, beta1, beta2, 1e-8, 0.01))
    W = [r.standard_normal((a, b), np.float32) for a, b in zip(dims, dims[1:])]
    net.set_params(W, [np.zeros(d, np.float32) for d in dims[1:]])
    net.upload_batch(r.standard_normal((batch, dims[0]), np.float32), r.standard_normal((batch, dims[-1]), np.float32))
    ctx.dispatch_forward(net.schedule)
    ctx.dispatch_loss(net.schedule, net.target)
    ctx.dispatch_backward(net.schedule)
    for call in (lambda: ctx.dispatch_optim(net.schedule), lambda: ctx.dispatch_optim(net.schedule),
                 lambda: ctx.dispatch_single_optim(net.schedule, net.W[0], 0)):
        with pytest.raises(FgError) as e:
            call()
        assert e.value.kind == "FG_ERR_INVALID_ARGUMENT"
        assert all(np.array_equal(a, b) for a, b in zip(net.get_params()[0], W))
    grads = {node: ctx.download(net.tensors.grad_tensors[i], np.empty(W[0].shape, np.float32))
             for i, node in enumerate(net.tensors.grad_nodes) if node == 1}      # (node 0 is the batch, 1 the first weights)
    good = _lib.AdamWHyper(lr, 0.9, 0.999, 1e-8, 0.01)
    ctx._check(ctx.lib.fg_exec_set_adamw(net.tensors.handle, C.byref(good)))
    ctx.dispatch_optim(net.schedule)
    ref, m, v = W[0].copy(), np.zeros_like(W[0]), np.zeros_like(W[0])
    oracle.adamw(ref, np.ascontiguousarray(grads[1]), m, v, lr, 0.9, 0.999, 1e-8, 0.01, 1)
    ok, worst = rel_err_ok(net.get_params()[0][0], ref, 1e-6)      # (as above)
    assert ok, f"{worst:.3g}"
    net.tensors.destroy()
    ctx.destroy()


def test_a_recorded_update_follows_the_hyperparameters():
    import ctypes as C

    from ferrograd_b200 import GpuContext, _lib
    from ferrograd_b200.mlp import GraphMLP
    dims, batch = [4, 8, 2], 16

    def train(plans):
        ctx = GpuContext(0)
        ctx.set_option("exec_plans", plans)
        r = np.random.Generator(np.random.Philox(5))
        net = GraphMLP(ctx, dims, batch, "tanh", "mse", ("adamw", 1e-2, 0.9, 0.999, 1e-8, 0.01))
        net.set_params([r.standard_normal((a, b), np.float32) for a, b in zip(dims, dims[1:])], [np.zeros(d, np.float32) for d in dims[1:]])
        net.upload_batch(r.standard_normal((batch, dims[0]), np.float32), r.standard_normal((batch, dims[-1]), np.float32))
        for step in range(6):
            if step == 3:      # (recorded in the second step, replayed from then on)
                hp = _lib.AdamWHyper(0.0, 0.5, 0.9, 1e-8, 0.3)
                ctx._check(ctx.lib.fg_exec_set_adamw(net.tensors.handle, C.byref(hp)))
            net.step()
        out = net.get_params()
        net.tensors.destroy()
        ctx.destroy()
        return out[0] + out[1]
    for a, b in zip(train("1"), train("0")):
        assert np.array_equal(a, b)
