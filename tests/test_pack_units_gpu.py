"""16-bit packs, sixteen slots a warp, and the windows beyond a pack that the tcgen05 kernel does not serve, against the dense restatement in float64."""
import pytest
import torch

from oracle import ssw_oracle as O
from tests.cases import rel_err
from tests.test_dense_streams_gpu import _boxes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("w,heads,hd,counts", [
    ((7, 7, 7), 3, 32, [1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64] * 2),
    ((7, 7, 7), 2, 16, [64, 65, 79, 80, 81, 343, 16, 1] * 2),   # beyond a pack: remainders of query and key blocks
    ((7, 7, 7), 12, 32, [16, 17, 12, 3] * 30),                  # packs of 32 slots; the table in global memory
    ((5, 6, 7), 1, 16, [9] * 1500),                             # more units than warps
    ((9, 9, 9), 6, 16, [729, 200, 40]),
])
def test_units(dtype, w, heads, hd, counts):
    from sparseswin3d_b200 import attention, window

    coords, dims = _boxes(counts, w, seed=heads)
    n = len(coords)
    g = torch.Generator().manual_seed(6)
    qkv = torch.randn(n, 3, heads, hd, generator=g).to(dtype)
    table = torch.randn((2 * w[0] - 1) * (2 * w[1] - 1) * (2 * w[2] - 1), heads, generator=g) * 0.5
    for shift in ((0, 0, 0), (w[0] // 2, 0, 0)):
        geom = window.resolve_geometry(1, dims, w, shift)
        plan = window.bucket_windows(coords=coords.cuda(), geom=geom, **attention.plan_params(heads, hd, dtype, w))
        out = attention.window_attention_fused(qkv.cuda(), plan, table.cuda(), hd ** -0.5, use_mask=bool(geom.shifted))
        plan.raise_on_error()
        idx = O.window_keys(coords, 1, dims, w, shift)[0]
        mask = O.compute_mask(tuple(geom.dims_p), tuple(geom.ws), tuple(geom.ss)) if geom.shifted else None
        ref = O.dense_window_attention(qkv.double(), idx, hd ** -0.5, table.double(), O.relative_position_index(w), mask)
        # one rounding of the output and that of the probabilities (bf16 keeps the rounding residual as well), which weigh values up to max |v|
        p_bits, o_bits = (2.0 ** -17, 2.0 ** -8) if dtype == torch.bfloat16 else (2.0 ** -11, 2.0 ** -11)
        bound = o_bits + p_bits * float(qkv[:, 2].double().abs().max() / ref.pow(2).mean().sqrt())
        assert rel_err(out.double().cpu(), ref) <= bound


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("c", [8, 40])   # one block of keys, several
def test_channels_are_added_up_in_order(dtype, c):
    """Sixteen consecutive channels a product: 2^24 + 1 is 2^24 in fp32, less 2^24 from channel 16 is 0, as a sum channel by channel gives it."""
    from sparseswin3d_b200 import attention, window

    w, hd = (7, 7, 7), 32
    coords, dims = _boxes([c] * 3, w, seed=1)
    n = len(coords)
    qkv = torch.zeros(n, 3, 1, hd)
    qkv[:, 0, 0, 0] = qkv[:, 0, 0, 16] = qkv[:, 1, 0, 0] = 4096.0
    qkv[:, 1, 0, 16] = -4096.0
    qkv[:, 0, 0, 1] = 1.0
    qkv[::2, 1, 0, 1] = 1.0   # every second key: with the 1 its score is 1
    qkv[::2, 2] = 1.0
    geom = window.resolve_geometry(1, dims, w, (0, 0, 0))
    plan = window.bucket_windows(coords=coords.cuda(), geom=geom, **attention.plan_params(1, hd, dtype, w))
    out = attention.window_attention_fused(qkv.to(dtype).cuda(), plan, torch.zeros(13 ** 3, 1).cuda(), 1.0, use_mask=False)
    plan.raise_on_error()
    win = O.window_keys(coords, 1, dims, w, (0, 0, 0))[0][:, 0]
    for x in win.unique():
        here = win == x
        # all scores 0: the mean of v, rounded to 16 bits
        assert (out.float().cpu()[here] - qkv[here, 2].mean(0)).abs().max() <= 2.0 ** -8


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("c, spoilt", [(16, 1), (20, 1), (4, 4)])   # a window a tile of sixteen slots, tiles of its own, four windows a tile
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("part", [1, 2])   # k, v
def test_rows_that_are_not_finite_spoil_their_tile_at_most(dtype, c, spoilt, value, part):
    from sparseswin3d_b200 import attention, window

    w, heads, hd = (7, 7, 7), 2, 32
    coords, dims = _boxes([c] * 40, w, seed=8)
    n = len(coords)
    qkv = torch.randn(n, 3, heads, hd, generator=torch.Generator().manual_seed(9)).to(dtype)
    table = torch.zeros(13 ** 3, heads, device="cuda")
    geom = window.resolve_geometry(1, dims, w, (0, 0, 0))
    plan = window.bucket_windows(coords=coords.cuda(), geom=geom, **attention.plan_params(heads, hd, dtype, w))
    whole = attention.window_attention_fused(qkv.cuda(), plan, table, hd ** -0.5, use_mask=False).cpu()
    qkv[17, part, 0] = value
    out = attention.window_attention_fused(qkv.cuda(), plan, table, hd ** -0.5, use_mask=False).cpu()
    plan.raise_on_error()
    win = O.window_keys(coords, 1, dims, w, (0, 0, 0))[0][:, 0]
    other = ~torch.isclose(out, whole, rtol=0, atol=0, equal_nan=True).view(n, -1).all(1)
    assert win[17] in win[other] and len(win[other].unique()) <= spoilt
    assert torch.equal(out.view(n, heads, hd)[:, 1], whole.view(n, heads, hd)[:, 1])   # (the other head is untouched)
