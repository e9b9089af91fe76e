"""fp32 GEMM with w kept in shared memory, at its longest sums and with several row tiles a block, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(40001, 96, 192), (40001, 96, 164), (20000, 288, 192), (19000, 20, 188), (40001, 96, 196)])
def test_kept_columns(m, n, k):
    from sparseswin3d_b200 import rows

    g = torch.Generator().manual_seed(k)
    x, w, b = torch.randn(m, k, generator=g).cuda(), torch.randn(n, k, generator=g).cuda(), torch.randn(n, generator=g).cuda()
    out = rows._gemm(x, w, b)
    ref = x.double() @ w.double().t() + b.double()
    err = out.double() - ref
    # 24 bits of each operand and chunks of 64 added up rounding to nearest: an ulp (2^-23) of the result, by its norm; a tile or a stage out of
    # place is of the result's size
    assert float(err.norm() / ref.norm()) <= 2.0 ** -22
    assert float(err.abs().max() / ref.square().mean().sqrt()) <= 2.0 ** -18
