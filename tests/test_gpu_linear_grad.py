"""The backward kernels of the sparse linear layer against 64-bit dense products, at the edges
of their tiles: row counts around the 64 / 128-row tiles and the four-row groups, k ranges and
column counts that leave the last tile ragged, contraction lengths that are cut into slices."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operand(pkg, N, K, n_keep, seed):
    W = K // 32 * n_keep
    DT = torch.from_numpy(pkg.formats.random_indices(seed, K, N // 32, n_keep)).cuda()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return torch.randn((W, N), device="cuda", generator=gen), DT, gen


def _check(pkg, M, N, K, n_keep, dtype, tol, want=(True, True)):
    values, DT, gen = _operand(pkg, N, K, n_keep, seed=M + N + K + n_keep)
    x = torch.randn((M, K), device="cuda", generator=gen).to(dtype)
    g = torch.randn((M, N), device="cuda", generator=gen).to(dtype)
    gx, gv = pkg.linear._sparse_grads(pkg, x, values, DT, n_keep, g, *want)
    torch.cuda.synchronize()
    assert pkg.device_status() == 0
    rows = pkg.linear._dense_rows(DT, n_keep)
    if want[0]:
        dense = torch.zeros((K, N), dtype=torch.float64, device="cuda").scatter_(0, rows, values.double())
        ref = g.double() @ dense.t()
        assert gx.dtype == dtype and float((gx.double() - ref).norm() / ref.norm()) <= max(tol, 1e-5)
    else:
        assert gx is None
    if want[1]:
        ref = (x.double().t() @ g.double()).gather(0, rows)
        assert gv.dtype == torch.float32 and float((gv.double() - ref).norm() / ref.norm()) <= 1e-5
    else:
        assert gv is None


@pytest.mark.parametrize("n_keep,K", [(16, 32), (16, 288), (12, 32), (12, 416), (8, 64), (8, 576), (4, 64), (4, 1088)])
@pytest.mark.parametrize("M,N", [(1, 32), (5, 160), (64, 128), (131, 416), (257, 1024)])
def test_gradients_at_tile_edges(pkg, M, N, K, n_keep):
    _check(pkg, M, N, K, n_keep, torch.float32, 1e-5)


@pytest.mark.parametrize("n_keep", [16, 12, 8, 4])
def test_gradients_of_long_contractions_in_slices(pkg, n_keep):
    _check(pkg, 3001, 256, 512, n_keep, torch.float32, 1e-5)       # few tiles of grad_B, many rows
    _check(pkg, 96, 8192, 256, n_keep, torch.float32, 1e-5)        # few tiles of grad_x, many columns
    _check(pkg, 2048, 2048, 2048, n_keep, torch.float32, 1e-5)     # whole tiles and a sliced rest


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 4e-3), (torch.float16, 5e-4)])      # one rounding of grad_x: 2^-9, 2^-12 at most per value
def test_gradients_in_16_bits(pkg, dtype, tol):
    for n_keep in (16, 12, 8, 4):
        _check(pkg, 77, 384, 320, n_keep, dtype, tol)


def test_one_gradient_at_a_time(pkg):
    _check(pkg, 70, 256, 256, 8, torch.float32, 1e-5, want=(True, False))
    _check(pkg, 70, 256, 256, 8, torch.float32, 1e-5, want=(False, True))


def test_backward_that_is_differentiated_again(pkg):
    torch.manual_seed(3)
    layer = pkg.linear.NMSparseLinear(pkg, torch.randn(128, 64, device="cuda"), 8)
    layer.values.requires_grad_(True)
    x = torch.randn(6, 64, device="cuda", requires_grad=True)
    (gx,) = torch.autograd.grad(layer(x).square().sum(), x, create_graph=True)
    (second,) = torch.autograd.grad(gx.square().sum(), layer.values)
    assert torch.isfinite(second).all() and float(second.norm()) > 0


def test_backward_is_an_operator(pkg):
    """Traced, compiled and batched backward passes reach the same kernels as a plain one."""
    from torch.fx.experimental.proxy_tensor import make_fx
    torch.manual_seed(4)
    layer = pkg.linear.NMSparseLinear(pkg, torch.randn(256, 128, device="cuda"), 8)
    layer.values.requires_grad_(True)
    x = torch.randn(8, 128, device="cuda", requires_grad=True)
    args = (x, layer.values, layer.op.D, layer.op.column_info, layer.raw_indices, 8, layer.op.format, layer.op.layout_ns, 32, 0)
    torch.library.opcheck(torch.ops.nmspmm_b200.sparse_linear, args)
    torch.library.opcheck(torch.ops.nmspmm_b200.sparse_linear_grad,
                          (x.detach(), layer.values.detach(), layer.raw_indices, torch.randn(8, 256, device="cuda"), 8, True, False))

    def step(x):
        x = x.detach().requires_grad_()
        return torch.autograd.grad(layer(x).square().sum(), (x, layer.values))

    want = step(x)
    for got in (make_fx(step)(x)(x), step(x)):
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    torch._dynamo.reset()
    xc = x.detach().clone().requires_grad_()
    torch.compile(lambda x: layer(x).square().sum(), backend="aot_eager")(xc).backward()
    assert torch.equal(xc.grad, want[0]) and torch.equal(layer.values.grad, want[1])
    y, c = layer(x), torch.randn(3, 8, 256, device="cuda")
    batched = torch.autograd.grad(y, (x, layer.values), c, is_grads_batched=True, retain_graph=True)
    for i in range(3):
        one = torch.autograd.grad(y, (x, layer.values), c[i], retain_graph=True)
        assert torch.equal(batched[0][i], one[0]) and torch.equal(batched[1][i], one[1])


def test_raw_indices_of_any_integer_type_and_stride(pkg):
    values, DT, gen = _operand(pkg, 256, 128, 8, seed=5)
    x, g = torch.randn((9, 128), device="cuda", generator=gen), torch.randn((9, 256), device="cuda", generator=gen)
    want = pkg.linear._sparse_grads(pkg, x, values, DT, 8, g, True, True)
    for raw in (DT.long(), DT.to(torch.uint8), DT.t().contiguous().t()):
        got = pkg.linear._sparse_grads(pkg, x, values, raw, 8, g, True, True)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
