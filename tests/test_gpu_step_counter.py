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
