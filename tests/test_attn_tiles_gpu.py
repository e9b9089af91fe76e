"""fp32 windows beyond a pack, against the dense restatement in float64: shares of query rows, key tiles, several units a block."""
import pytest
import torch

from oracle import ssw_oracle as O
from tests.cases import rel_err
from tests.test_dense_streams_gpu import _boxes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,heads,hd,counts", [
    ((7, 7, 7), 6, 32, [343, 25, 24, 64, 65, 96, 97, 128, 129, 192, 193] * 3),   # packs of 24 rows
    ((7, 7, 7), 12, 32, [70, 9, 8, 100] * 2),          # packs of 8 rows
    ((7, 7, 7), 3, 32, [49, 48, 47, 65, 200] * 2),     # packs of 48 rows
    ((10, 10, 10), 6, 16, [1000, 961, 40]),            # sixteen shares
    ((7, 7, 7), 24, 16, [50] * 60),                    # more units than blocks
    ((7, 7, 7), 12, 32, [20] * 850 + [3] * 10),        # packs of 16 rows, and windows beyond them too small on average
    ((7, 7, 7), 12, 32, [20] * 200 + [40] * 330),      # ... and not
])
def test_windows_beyond_a_pack(w, heads, hd, counts):
    from sparseswin3d_b200 import attention, window

    coords, dims = _boxes(counts, w, seed=heads)
    n = len(coords)
    g = torch.Generator().manual_seed(4)
    qkv = torch.randn(n, 3, heads, hd, generator=g)
    table = torch.randn((2 * w[0] - 1) * (2 * w[1] - 1) * (2 * w[2] - 1), heads, generator=g)
    for shift in ((0, 0, 0), (w[0] // 2, 0, 0)):
        geom = window.resolve_geometry(1, dims, w, shift)
        plan = window.bucket_windows(coords=coords.cuda(), geom=geom, **attention.plan_params(heads, hd, torch.float32, w))
        out = attention.window_attention_fused(qkv.cuda(), plan, table.cuda(), hd ** -0.5, use_mask=bool(geom.shifted))
        plan.raise_on_error()
        idx = O.window_keys(coords, 1, dims, w, shift)[0]
        mask = O.compute_mask(tuple(geom.dims_p), tuple(geom.ws), tuple(geom.ss)) if geom.shifted else None
        ref = O.dense_window_attention(qkv, idx, hd ** -0.5, table, O.relative_position_index(w), mask)
        # scores up to some tens carry a few ulp (2^-24 each) into the exponent; sums of up to 1000 terms in chunks
        assert rel_err(out.double().cpu(), ref) <= 1e-5
