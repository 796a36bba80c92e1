"""The input gradient's larger register tiles: sizes past the line from which they are taken that leave the last tile
of rows and of k ragged, few vectors per group of warps, slices, 16-bit operands.  Against 64-bit dense products;
1e-5 as in test_gpu_linear_grad.py (sums of up to 5500 products in 32 bits, 5e-7 seen), one rounding more in 16 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,n_keep", [(777, 2080, 1120, 16), (1001, 2080, 1120, 12), (1501, 2080, 1088, 8),       # everything ragged
                                          (5003, 160, 2048, 16), (9001, 224, 1024, 12), (9001, 96, 4096, 8),            # 3 to 7 vectors
                                          (131, 11008, 1184, 16), (130, 16384, 992, 12), (258, 12288, 1024, 8)])        # few tiles: slices
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 4e-3)])
def test_input_gradient(pkg, M, N, K, n_keep, dtype, tol):
    W = K // 32 * n_keep
    assert M * N * W >= 7.4e8
    DT = torch.from_numpy(pkg.formats.random_indices(M, K, N // 32, n_keep)).cuda()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M + n_keep)
    values = torch.randn((W, N), device="cuda", generator=gen)
    x = torch.randn((M, K), device="cuda", generator=gen).to(dtype)
    g = torch.randn((M, N), device="cuda", generator=gen).to(dtype)
    gx, none = pkg.linear._sparse_grads(pkg, x, values, DT, n_keep, g, True, False)
    again, _ = pkg.linear._sparse_grads(pkg, x, values, DT, n_keep, g, True, False)
    assert none is None and gx.dtype == dtype and torch.equal(gx, again) and pkg.device_status() == 0
    dense = torch.zeros((K, N), dtype=torch.float64, device="cuda").scatter_(0, pkg.linear._dense_rows(DT, n_keep), values.double())
    ref = g.double() @ dense.t()
    assert float((gx.double() - ref).norm() / ref.norm()) <= tol


def test_more_rows_than_a_grid_has_blocks_along_y(pkg):
    """The transposing pass over grad_y cuts the rows into blocks of 32, of which a grid holds 65535 along y."""
    M, N, K, n_keep = 65535 * 32 + 100, 32, 64, 8
    DT = torch.from_numpy(pkg.formats.random_indices(1, K, N // 32, n_keep)).cuda()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    values, g = torch.randn((K // 32 * n_keep, N), device="cuda", generator=gen), torch.randn((M, N), device="cuda", generator=gen)
    assert M * N * values.shape[0] >= 7.4e8
    gx, _ = pkg.linear._sparse_grads(pkg, torch.empty((M, K), device="cuda"), values, DT, n_keep, g, True, False)
    dense = torch.zeros((K, N), dtype=torch.float64, device="cuda").scatter_(0, pkg.linear._dense_rows(DT, n_keep), values.double())
    ref = g.double() @ dense.t()
    for rows in (slice(0, 1 << 20), slice(1 << 20, 65535 * 32), slice(65535 * 32, M)):
        assert float((gx[rows].double() - ref[rows]).norm() / ref[rows].norm()) <= 1e-5
    assert pkg.device_status() == 0
