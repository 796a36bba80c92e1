"""The input gradient's larger register tiles: sizes at which they are taken that leave the last tile
of rows and of k ragged, few vectors per group of warps, slices, 16-bit operands.  Against 64-bit dense products;
1e-5 as in test_gpu_linear_grad.py (sums of up to 5500 products in 32 bits, 5e-7 seen), one rounding more in 16 bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def takes_larger_tiles(pkg, M, N, K, n_keep):
    """The workspace then holds both transposed operands beside the slices' slots of 128 x 256 floats."""
    d = pkg.make_desc(M, N, K, n_keep, pkg.FORMAT_LOW, 32)
    need = pkg.load_library().nmspmm_linear_grad_workspace_bytes(ctypes.byref(d), pkg.DTYPE_F32, 1, 0) - 256
    copies = 4 * N * ((M + 3) // 4 * 4 + (K // 32 * n_keep + 3) // 4 * 4)
    assert copies % (128 * 256 * 4) >= 256
    return (need - copies) % (128 * 256 * 4) < 256


@pytest.mark.parametrize("M,N,K,n_keep", [(777, 2080, 1120, 16), (1001, 2080, 1120, 12), (1501, 2080, 1088, 8),       # everything ragged
                                          (5003, 160, 2048, 16), (9001, 224, 2016, 12), (9001, 96, 4096, 8),            # 3 to 7 vectors
                                          (131, 11008, 1184, 16), (130, 16352, 1504, 12), (258, 12288, 1024, 8)])        # few tiles: slices
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 4e-3)])
def test_input_gradient(pkg, M, N, K, n_keep, dtype, tol):
    W = K // 32 * n_keep
    assert takes_larger_tiles(pkg, M, N, K, n_keep)
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
    M, N, K, n_keep = 65535 * 32 + 100, 32, 512, 16
    DT = torch.from_numpy(pkg.formats.random_indices(1, K, N // 32, n_keep)).cuda()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    values, g = torch.randn((K // 32 * n_keep, N), device="cuda", generator=gen), torch.randn((M, N), device="cuda", generator=gen)
    assert takes_larger_tiles(pkg, M, N, K, n_keep)
    gx, _ = pkg.linear._sparse_grads(pkg, torch.empty((M, K), device="cuda"), values, DT, n_keep, g, True, False)
    dense = torch.zeros((K, N), dtype=torch.float64, device="cuda").scatter_(0, pkg.linear._dense_rows(DT, n_keep), values.double())
    for rows in (slice(0, 1 << 20), slice(1 << 20, 65535 * 32), slice(65535 * 32, M)):
        ref = g[rows].double() @ dense.t()
        assert float((gx[rows].double() - ref).norm() / ref.norm()) <= 1e-5
    assert pkg.device_status() == 0


@pytest.mark.parametrize("M,N,K,n_keep,larger", [(2049, 4064, 4096, 8, True), (256, 4160, 4096, 8, True), (128, 4160, 4096, 8, False),
                                                 (100, 4224, 4992, 12, False), (128, 17792, 9920, 16, False),
                                                 (1315, 10112, 5824, 8, True)])
def test_where_they_are_taken(pkg, M, N, K, n_keep, larger):
    assert takes_larger_tiles(pkg, M, N, K, n_keep) == larger
