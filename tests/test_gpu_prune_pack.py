"""Pruning and packing in one pass against the two steps apart: the same kept values, packed indices and lists, bit for bit,
for every ratio and format, odd numbers of windows, ties and values that are not numbers."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_keep,fmt", [(32, 0), (16, 0), (12, 0), (8, 0), (8, 1), (4, 1)])
@pytest.mark.parametrize("K,N", [(64, 128), (320, 640), (1088, 384), (96, 256)])
@pytest.mark.parametrize("vec_len", [32, 64])
@pytest.mark.parametrize("values", ["random", "ties", "not_finite"])
def test_same_as_apart(pkg, n_keep, fmt, K, N, vec_len, values):
    if fmt == pkg.FORMAT_HIGH and K % 64:
        pytest.skip("windows come in pairs")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(K + N + n_keep)
    dense = torch.randn((K, N), device="cuda", generator=gen)
    if values == "ties":
        dense = dense.sign() * 0.5                               # every row's score is the same
    if values == "not_finite":
        dense[::7, ::5], dense[3::11, 2::9], dense[5::13, ::17] = float("nan"), float("inf"), float("-inf")
    op = pkg.NMSpMM.from_dense(dense, n_keep, vec_len, fmt=fmt)
    BT, DT = pkg.prune_device(dense, n_keep, vec_len)
    apart = pkg.NMSpMM(BT, DT, K, n_keep, fmt=fmt, vec_len=vec_len)
    assert torch.equal(op.B.view(torch.int32), BT.view(torch.int32)) and torch.equal(op.D, apart.D)
    assert (op.column_info is None) == (apart.column_info is None)
    if op.column_info is not None:
        assert torch.equal(op.column_info, apart.column_info)
    assert (op.K, op.N, op.W, op.n_keep, op.format, op.layout_ns, op.vec_len) == (apart.K, apart.N, apart.W, apart.n_keep, apart.format,
                                                                                 apart.layout_ns, apart.vec_len)
    if values == "random":
        A = torch.randn((K, 8), device="cuda", generator=gen)
        assert torch.equal(op.matmul(A), apart.matmul(A))


def test_what_one_pass_does_not_take_goes_the_two_step_way(pkg):
    dense = torch.randn((128, 256), device="cuda")
    for n_keep in (0, 33):
        with pytest.raises(pkg.NMSpMMError) as e:
            pkg.NMSpMM.from_dense(dense, n_keep, fmt=pkg.FORMAT_HIGH)
        assert e.value.status == pkg.INVALID_ARGUMENT
    other = pkg.NMSpMM.from_dense(dense, 8, fmt=2)               # no format of the multiply: packed as the 32-k one
    assert torch.equal(other.D, pkg.NMSpMM.from_dense(dense, 8, fmt=pkg.FORMAT_LOW).D) and other.format == 2
