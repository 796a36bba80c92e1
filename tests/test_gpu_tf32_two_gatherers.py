"""Two gathering threads on an odd number of stages: a thread meets a stage every second time round, so its wait for
the stage has to be unmistakable when the step between is still being filled.  And 16-bit rows, whose steps go to the
products in pairs.  Long contractions in few tiles, many calls: every call gives the first one's bits, within TF32 of the
oracle (10 mantissa bits of both operands: 2e-3; one rounding of a bfloat16 result more: 7e-3)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_keep,vec_len,tile", [(12, 64, 5), (16, 64, 5), (8, 32, 12), (12, 32, 12), (16, 32, 12)])
@pytest.mark.parametrize("M,N", [(16, 1216), (128, 4864)])
def test_repeated_calls(pkg, orc, n_keep, vec_len, tile, M, N):
    N = N // 192 * 192 + vec_len
    p = pkg.formats.make_random(M, N, 10560, n_keep, vec_len=vec_len, seed=n_keep + M)
    op = pkg.NMSpMM.from_problem(p, layout_ns=vec_len, fmt=0)
    A = torch.from_numpy(p.A_km).cuda()
    first = op.matmul(A, path=pkg.PATH_TF32, tile=tile)
    want = orc.nm_gemm_f64(p.A_km, p.B_col, p.D_col)
    err = float(np.linalg.norm(first.double().cpu().numpy() - want) / np.linalg.norm(want))
    assert err <= 2e-3
    for _ in range(20):
        assert torch.equal(op.matmul(A, path=pkg.PATH_TF32, tile=tile), first)
    assert pkg.device_status() == 0


@pytest.mark.parametrize("n_keep,fmt,vec_len,tile", [(8, 0, 32, 12), (8, 1, 32, 12), (4, 1, 32, 12), (8, 1, 64, 5), (4, 1, 64, 5)])
@pytest.mark.parametrize("M,N", [(16, 1216), (129, 4864)])
@pytest.mark.parametrize("dtype,tol", [(torch.float16, 2e-3), (torch.bfloat16, 7e-3)])
def test_repeated_calls_on_pairs_of_steps(pkg, orc, n_keep, fmt, vec_len, tile, M, N, dtype, tol):
    N = N // 192 * 192 + vec_len
    p = pkg.formats.make_random(M, N, 10560, n_keep, vec_len=vec_len, seed=n_keep + M)       # 330 steps (165 at 4:32: an odd one at the end)
    op = pkg.NMSpMM.from_problem(p, layout_ns=vec_len, fmt=fmt)
    x = torch.from_numpy(p.A_km).cuda().t().contiguous().to(dtype)
    first = op.matmul_rows(x, path=pkg.PATH_TF32, tile=tile)
    want = orc.nm_gemm_f64(x.float().t().contiguous().cpu().numpy(), p.B_col, p.D_col)
    assert float(np.linalg.norm(first.double().cpu().numpy() - want) / np.linalg.norm(want)) <= tol
    for _ in range(20):
        assert torch.equal(op.matmul_rows(x, path=pkg.PATH_TF32, tile=tile), first)
    assert pkg.device_status() == 0
