"""Two gathering threads on an odd number of stages: a thread meets a stage every second time round, so its wait for
the stage has to be unmistakable when the step between is still being filled.  Long contractions in few tiles, many
calls: every call gives the first one's bits, within TF32 of the oracle (10 mantissa bits of both operands: 2e-3)."""
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
