"""The sparse linear operator as torch sees it, on the CPU: a dense stand-in takes the place of the two
kernels, so that what is checked is the registration and the autograd formula -- tracing, compiling
and batching a backward pass through it."""
import pytest
import torch

N_KEEP, M, K, N = 8, 6, 64, 128


@pytest.fixture(scope="module")
def op(pkg_host):
    linear = pkg_host.linear
    linear.register_ops(pkg_host)

    def dense(x, values, raw):
        return torch.zeros(x.shape[1], values.shape[1]).scatter_(0, linear._dense_rows(raw, N_KEEP), values)

    def forward(x, values, packed, column_info, raw, n_keep, fmt, layout_ns, vec_len, path):
        return x @ dense(x, values, raw)

    def grads(x, values, raw, grad_y, n_keep, want_x, want_values):
        rows = linear._dense_rows(raw, n_keep)
        return (grad_y @ dense(x, values, raw).t() if want_x else x.new_empty(0),
                (x.t() @ grad_y).gather(0, rows) if want_values else values.new_empty(0))

    stand_in = torch.library.Library("nmspmm_b200", "IMPL")
    stand_in.impl("sparse_linear", forward, "CPU")
    stand_in.impl("sparse_linear_grad", grads, "CPU")
    yield torch.ops.nmspmm_b200.sparse_linear
    del stand_in


@pytest.fixture(scope="module")
def operand(pkg_host):
    torch.manual_seed(1)
    raw = torch.from_numpy(pkg_host.formats.random_indices(3, K, N // 32, N_KEEP))
    return torch.randn(M, K), torch.randn(raw.shape[0], N), raw


def _apply(op, x, values, raw):
    return op(x, values, torch.zeros(4, dtype=torch.int32), None, raw, N_KEEP, 1, 128, 32, 0)


def _step(op, raw):
    def step(x, values):
        x, values = x.detach().requires_grad_(), values.detach().requires_grad_()
        return torch.autograd.grad(_apply(op, x, values, raw).square().sum(), (x, values))
    return step


def _close(got, want):
    assert len(got) == len(want)
    for g, w in zip(got, want):
        assert g.shape == w.shape and float((g - w).norm() / w.norm()) <= 1e-5


def test_a_traced_training_step_holds_the_gradients(op, operand):
    from torch.fx.experimental.proxy_tensor import make_fx
    x, values, raw = operand
    step = _step(op, raw)
    graph = make_fx(step)(x, values)
    assert any(n.target is torch.ops.nmspmm_b200.sparse_linear_grad.default for n in graph.graph.nodes)
    other = torch.randn(M, K)
    _close(graph(other, values), step(other, values))


@pytest.mark.parametrize("dynamic", [False, True])
def test_a_compiled_training_step(op, operand, dynamic):
    x, values, raw = operand
    torch._dynamo.reset()
    xc, vc = x.clone().requires_grad_(), values.clone().requires_grad_()
    loss = torch.compile(lambda x, v: _apply(op, x, v, raw).square().sum(), backend="aot_eager", dynamic=dynamic, fullgraph=True)
    loss(xc, vc).backward()
    _close((xc.grad, vc.grad), _step(op, raw)(x, values))


@pytest.mark.parametrize("wanted", [(True, True), (True, False), (False, True)])
def test_batched_cotangents(op, operand, wanted):
    x, values, raw = operand
    x, values = x.clone().requires_grad_(wanted[0]), values.clone().requires_grad_(wanted[1])
    inputs = [t for t in (x, values) if t.requires_grad]
    y = _apply(op, x, values, raw)
    cotangents = torch.randn(3, M, N)
    batched = torch.autograd.grad(y, inputs, cotangents, is_grads_batched=True, retain_graph=True)
    one_by_one = zip(*[torch.autograd.grad(y, inputs, c, retain_graph=True) for c in cotangents])
    _close(batched, [torch.stack(g) for g in one_by_one])


def test_backward_on_meta_tensors(op, operand):
    x, values, raw = (t.to("meta") for t in operand)
    x.requires_grad_()
    values.requires_grad_()
    y = op(x, values, torch.zeros(4, dtype=torch.int32, device="meta"), None, raw, N_KEEP, 1, 128, 32, 0)
    gx, gv = torch.autograd.grad(y.sum(), (x, values))
    assert gx.shape == x.shape and gv.shape == values.shape


def test_a_second_copy_of_the_package_shares_the_operator(op, pkg_host):
    import importlib.util
    import os
    import sys
    here = os.path.dirname(pkg_host.__file__)
    spec = importlib.util.spec_from_file_location("nm_spmm_second", os.path.join(here, "__init__.py"), submodule_search_locations=[here])
    second = importlib.util.module_from_spec(spec)
    sys.modules["nm_spmm_second"] = second
    try:
        spec.loader.exec_module(second)
        assert second.linear.register_ops(second) is pkg_host.linear.register_ops(pkg_host)
    finally:
        for name in [n for n in sys.modules if n.split(".")[0] == "nm_spmm_second"]:
            del sys.modules[name]


@pytest.mark.parametrize("allowed,rows,kernels", [(False, 4096, True), (True, 4096, False), (True, 128, True)])
def test_large_backward_follows_torchs_tf32_switch(op, pkg_host, allowed, rows, kernels):
    """With TF32 products allowed a large backward is faster on torch's dense ones; otherwise it takes the kernels."""
    from torch.fx.experimental.proxy_tensor import make_fx
    size, raw = 4096, torch.zeros(4096 // 32 * N_KEEP, 4096 // 32, dtype=torch.int32, device="meta")

    def step(x, values):
        x, values = x.detach().requires_grad_(), values.detach().requires_grad_()
        y = op(x, values, torch.zeros(4, dtype=torch.int32, device="meta"), None, raw, N_KEEP, 1, 128, 32, 0)
        return torch.autograd.grad(y.square().sum(), (x, values))

    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = allowed
    try:
        graph = make_fx(step)(torch.empty(rows, size, device="meta"), torch.empty(size // 32 * N_KEEP, size, device="meta"))
    finally:
        torch.backends.cuda.matmul.allow_tf32 = before
    called = [n.target for n in graph.graph.nodes]
    assert (torch.ops.nmspmm_b200.sparse_linear_grad.default in called) == kernels
    assert (torch.ops.aten.mm.default in called) != kernels
