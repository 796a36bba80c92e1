"""The tensor-core path's 192-column tiles: six vectors a tile (so a tile starts inside an index block), a last tile
with fewer, ragged rows, an odd number of steps, K slices, every way A is read, C in the type of A.  Tolerances as in
test_gpu_tf32.py: 10 mantissa bits of FP32 operands (7e-4 seen), one rounding of a 16-bit result."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TILE = 12


@pytest.mark.parametrize("n_keep,fmt,K", [(16, 0, 544), (12, 0, 608), (8, 0, 352), (8, 1, 576), (4, 1, 704)])
@pytest.mark.parametrize("M,N,layout", [(4, 192, 32), (136, 576, 64), (260, 640, 128), (129, 544, 32)])
@pytest.mark.parametrize("kind", ["cols", "f32", "f16", "bf16"])
@pytest.mark.parametrize("split_k", [0, 1, 3])
def test_edges(pkg, orc, n_keep, fmt, K, M, N, layout, kind, split_k):
    if kind == "cols" and M % 4:
        pytest.skip("col-major A starts every k row on 16 bytes")
    p = pkg.formats.make_random(M, N, K, n_keep, seed=M + N + K)
    op = pkg.NMSpMM.from_problem(p, layout_ns=layout, fmt=fmt)
    A = torch.from_numpy(p.A_km).cuda()
    if kind == "cols":
        got, tol = op.matmul(A, path=pkg.PATH_TF32, tile=TILE, split_k=split_k), 2e-3
    else:
        dtype = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[kind]
        x = A.t().contiguous().to(dtype)
        got, tol = op.matmul_rows(x, path=pkg.PATH_TF32, tile=TILE, split_k=split_k), (7e-3 if kind == "bf16" else 2e-3)
        assert got.dtype == dtype
        A = x.float().t().contiguous()
    want = orc.nm_gemm_f64(A.cpu().numpy(), p.B_col, p.D_col)
    err = float(np.linalg.norm(got.double().cpu().numpy() - want) / np.linalg.norm(want))
    assert err <= tol and pkg.device_status() == 0


def test_a_call_takes_them_where_they_leave_fewer_sms_idle(pkg):
    p = pkg.formats.make_random(256, 11008, 1024, 16, seed=2)
    op = pkg.NMSpMM.from_problem(p)
    d = op.desc(256, path=pkg.PATH_TF32)
    assert pkg.plan(d).tile == pkg.TILE_128x256 and pkg.call_plan(d).tile == TILE
    A = torch.from_numpy(p.A_km).cuda()
    got, other = op.matmul(A, path=pkg.PATH_TF32), op.matmul(A, path=pkg.PATH_TF32, tile=5)
    assert torch.equal(got, other)                             # whole tiles either way: the same products in the same order
