"""The wide tiles of the exact path (128 x 256, 256 x 128, 64 x 512) at the edges of their tiles and
rings: ragged rows, vectors past the last column, fewer windows than stages, pieces that cross tiles,
every index layout, and the call that picks them by itself.  Against the oracle's float product; 1e-5 as for
the other exact kernels (32-bit sums of up to 1024 products, 8e-7 seen)."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TILES = (5, 10, 11)
TOL = 1e-5


def rel_err(got, want):
    return float(np.linalg.norm(got.astype(np.float64) - want.astype(np.float64)) / np.linalg.norm(want.astype(np.float64)))


@pytest.mark.parametrize("tile", TILES)
@pytest.mark.parametrize("n_keep,fmt,K", [(16, 0, 96), (12, 0, 608), (32, 0, 160), (8, 0, 320), (8, 1, 640), (4, 1, 1088), (8, 1, 64)])
@pytest.mark.parametrize("M,N,layout", [(4, 32, 32), (68, 288, 32), (256, 576, 64), (260, 640, 128)])
@pytest.mark.parametrize("split_k", [0, 1, 2, 7])
def test_edges(pkg, orc, tile, n_keep, fmt, K, M, N, layout, split_k):
    p = pkg.formats.make_random(M, N, K, n_keep, seed=M + N + K)
    want = orc.nm_gemm_f32(p.A_km, p.B_col, p.D_col)
    op = pkg.NMSpMM.from_problem(p, layout_ns=layout, fmt=fmt)
    A = torch.from_numpy(p.A_km).cuda()
    C = torch.full((M, N), float("nan"), device="cuda")
    op.matmul(A, tile=tile, split_k=split_k, out=C)
    assert rel_err(C.cpu().numpy(), want) <= TOL
    assert torch.equal(op.matmul(A, tile=tile, split_k=split_k), C)      # one order of sums
    assert pkg.device_status() == 0


@pytest.mark.parametrize("M,N,K,n_keep", [(776, 2560, 2080, 12), (1024, 5760, 1024, 12), (2048, 5760, 1024, 16), (64, 11008, 4096, 8), (128, 1024, 65536, 4), (2048, 1152, 4096, 16)])
def test_calls_that_take_a_wide_tile_by_themselves(pkg, M, N, K, n_keep):
    """Whatever scratch the call is handed: the wide tile where its pieces fit, the planned one otherwise.
    Row-major callers and several outputs take the same route."""
    p = pkg.formats.make_random(M, N, K, n_keep, seed=9)
    op = pkg.NMSpMM.from_problem(p)
    A = torch.from_numpy(p.A_km).cuda()
    d = op.desc(M)
    named, taken, own = pkg.plan(d).tile, pkg.call_plan(d).tile, pkg.workspace_bytes(d)
    fits = pkg.workspace_bytes(op.desc(M, tile=taken)) <= own
    assert taken in TILES and pkg.call_plan(d, own).tile == (taken if fits else named)
    planned = op.matmul(A, tile=named)
    got = op.matmul(A)
    small = torch.zeros(max(own, 16), dtype=torch.uint8, device="cuda")
    with_less = torch.empty_like(got)
    pkg.gemm(d, A, op.B, op.D, op.column_info, with_less, small)
    assert torch.equal(got, op.matmul(A, tile=taken)) and torch.equal(with_less, got if fits else planned)
    rows = op.matmul_rows(A.t().contiguous())
    wide_buffer = torch.full((2, M, N + 64), -1.0, device="cuda")
    op.matmul_into(A, [wide_buffer[0].data_ptr(), wide_buffer[1].data_ptr()], N + 64, 32)
    for other in (got, with_less, rows, wide_buffer[0][:, 32:-32], wide_buffer[1][:, 32:-32]):
        assert float((other.double() - planned.double()).norm() / planned.double().norm()) <= TOL
    assert bool((wide_buffer[:, :, :32] == -1).all()) and bool((wide_buffer[:, :, -32:] == -1).all())
    assert pkg.device_status() == 0


@pytest.mark.parametrize("M,N,K,n_keep,path", [(2048, 5760, 1024, 16, 0), (2052, 5760, 1024, 8, 0), (512, 11008, 1024, 12, 0),
                                               (132, 1024, 1024, 16, 1), (256, 1024, 1024, 12, 1)])
def test_row_major_calls_with_the_named_plans_scratch(pkg, M, N, K, n_keep, path):
    """Scratch for the plan that the description names and not a byte more: that plan runs, bit for bit."""
    p = pkg.formats.make_random(M, N, K, n_keep, seed=19)
    op = pkg.NMSpMM.from_problem(p)
    d, x = op.desc(M, path=path), torch.from_numpy(p.A_km).cuda().t().contiguous()
    own = pkg.workspace_bytes(d)
    assert own < pkg.call_workspace_bytes(d) and pkg.call_plan(d, own).tile == pkg.plan(d).tile
    less = max(own, 64 << 10) + (0 if path == pkg.PATH_TF32 else 4 * M * K)
    got, ws = torch.full((M, N), float("nan"), device="cuda"), torch.zeros(less, dtype=torch.uint8, device="cuda")
    rc = pkg.load_library().nmspmm_gemm_row_major(
        ctypes.byref(d), x.data_ptr(), op.B.data_ptr(), op.D.data_ptr(), None if op.column_info is None else op.column_info.data_ptr(),
        got.data_ptr(), ws.data_ptr(), less, torch.cuda.current_stream().cuda_stream)
    assert rc == pkg.OK and torch.equal(got, op.matmul_rows(x, path=path, tile=pkg.plan(d).tile)) and pkg.device_status() == 0


def test_non_finite_values_stay_where_they_belong(pkg):
    """An infinity or a NaN in A reaches the columns whose lists name its k, and no other."""
    p = pkg.formats.make_random(256, 1024, 1024, 8, seed=3)
    op = pkg.NMSpMM.from_problem(p)
    A = torch.from_numpy(p.A_km).cuda()
    A[5, 7], A[70, 200] = float("inf"), float("nan")
    for tile in TILES:
        assert torch.equal(torch.isfinite(op.matmul(A, tile=tile)), torch.isfinite(op.matmul(A, tile=1)))


@pytest.mark.parametrize("tile", TILES)
def test_a_wait_that_runs_out_is_reported(pkg, tile):
    """As in test_gpu_timeout.py: stages that never fill, nothing stored, usable afterwards."""
    p = pkg.formats.make_random(128, 512, 1024, 8, seed=301)
    op = pkg.NMSpMM.from_problem(p)
    A = torch.from_numpy(p.A_km).cuda()
    want = op.matmul(A, tile=1)
    for split_k in (1, 2):
        C = torch.full((128, 512), 7.0, device="cuda")
        assert pkg.test_short_fill(True) == 0
        try:
            op.matmul(A, tile=tile, split_k=split_k, out=C)
            torch.cuda.synchronize()
        finally:
            pkg.test_short_fill(False)
        assert bool((C == 7.0).all())
        assert pkg.load_library().nmspmm_device_status(None, 1) == pkg.DEVICE_TIMEOUT
        got = op.matmul(A, tile=tile, split_k=split_k)
        assert float((got - want).norm() / want.norm()) <= TOL and pkg.device_status() == 0
