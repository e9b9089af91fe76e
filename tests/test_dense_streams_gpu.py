"""Windows beyond a pack, 16-bit: two query tiles in flight over a ring of key tiles, and the layouts of the bias slice, against the
dense restatement in float64."""
import pytest
import torch

from oracle import ssw_oracle as O
from tests.cases import rel_err

pytestmark = pytest.mark.gpu


def _boxes(counts, w, seed):
    """One window w per entry of `counts`, side by side, that many voxels in it, listed in random order."""
    g = torch.Generator().manual_seed(seed)
    n, rows = w[0] * w[1] * w[2], []
    for k, c in enumerate(counts):
        pos = torch.randperm(n, generator=g)[:c]
        rows.append(torch.stack([torch.zeros_like(pos), k * w[0] + pos // (w[1] * w[2]), pos // w[2] % w[1], pos % w[2]], 1))
    coords = torch.cat(rows).int()
    return coords[torch.randperm(len(coords), generator=g)].contiguous(), (len(counts) * w[0], w[1], w[2])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("w,heads,counts", [
    ((7, 7, 7), 3, [343, 65, 66, 96, 97, 128, 129, 192, 193, 256, 257, 288, 289] * 12),  # units of one to three query tiles, one to four key tiles
    ((7, 7, 7), 5, [100] * 70),          # one query tile a unit: a stream without work in every other one; 145 blocks
    ((9, 9, 9), 2, [729, 70, 385, 384, 640, 641] * 4),
    ((8, 8, 8), 20, [512, 80] * 2),      # 140 blocks
    ((6, 6, 6), 15, [216, 100] * 12),    # 135 blocks would leave out one in eleven: all of them, changing heads
    ((2, 16, 31), 2, [992, 961, 100]),   # one query tile buffer a stream, eleven key tiles
    ((22, 23, 2), 1, [1012, 500, 90]),   # a padded bias slice would not fit
    ((9, 9, 11), 3, [891, 300]),
])
def test_window_mixes(dtype, w, heads, counts):
    from sparseswin3d_b200 import attention, window

    hd = 32
    coords, dims = _boxes(counts, w, seed=len(counts))
    n = len(coords)
    g = torch.Generator().manual_seed(3)
    qkv = torch.randn(n, 3, heads, hd, generator=g).to(dtype)
    table = torch.randn((2 * w[0] - 1) * (2 * w[1] - 1) * (2 * w[2] - 1), heads, generator=g) * 0.5
    shift = tuple(x // 2 if d > x else 0 for x, d in zip(w, dims)) if heads == 3 else (0, 0, 0)
    geom = window.resolve_geometry(1, dims, w, shift)
    plan = window.bucket_windows(coords=coords.cuda(), geom=geom, **attention.plan_params(heads, hd, dtype, w))
    out = attention.window_attention_fused(qkv.cuda(), plan, table.cuda(), hd ** -0.5, use_mask=bool(geom.shifted))
    plan.raise_on_error()
    idx = O.window_keys(coords, 1, dims, w, shift)[0]
    mask = O.compute_mask(tuple(geom.dims_p), tuple(geom.ws), tuple(geom.ss)) if geom.shifted else None
    ref = O.dense_window_attention(qkv.double(), idx, hd ** -0.5, table.double(), O.relative_position_index(w), mask)
    # one rounding of the output (2^-8 / 2^-11 of it at most) and that of the probabilities (2^-17; fp16 2^-11: the packs' kernel), which
    # weigh values up to max |v|, over the rms the error is measured by
    p_bits, o_bits = (2.0 ** -17, 2.0 ** -8) if dtype == torch.bfloat16 else (2.0 ** -11, 2.0 ** -11)
    bound = o_bits + p_bits * float(qkv[:, 2].double().abs().max() / ref.pow(2).mean().sqrt())
    assert rel_err(out.double().cpu(), ref) <= bound


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_key_tiles_beyond_the_bound_are_added_up_rounding_to_nearest(dtype):
    """All weights 1, a value of 2^14 in the first key tile and of -2^14 in the last, 2^-14 in those between: a tile's 96 of these are
    three units in the last place of 2^14 together, which fp32 adds keep and sums that are cut off product by product lose."""
    from sparseswin3d_b200 import attention, window

    w, heads, hd = (9, 9, 9), 2, 32
    coords, dims = _boxes([729, 729], w, seed=2)
    n = len(coords)
    geom = window.resolve_geometry(1, dims, w, (0, 0, 0))
    plan = window.bucket_windows(coords=coords.cuda(), geom=geom, **attention.plan_params(heads, hd, dtype, w))
    at = O.window_keys(coords, 1, dims, w, (0, 0, 0))[0][:, 1].long()   # full windows: keys come by position
    v = torch.zeros(729)
    v[96:672] = 2.0 ** -14
    v[3], v[700] = 2.0 ** 14, -(2.0 ** 14)
    qkv = torch.zeros(n, 3, heads, hd, dtype=dtype)
    qkv[:, 2] = v[at].to(dtype)[:, None, None]
    # a bias beyond the bound for one pair of the window, the query in one corner and the key in the other
    table = torch.zeros(17 ** 3, heads)
    table[-1] = 100.0
    out = attention.window_attention_fused(qkv.cuda(), plan, table.cuda(), hd ** -0.5, use_mask=False).float().cpu()
    plan.raise_on_error()
    exact = 576 * 2.0 ** -14 / 729
    rest = at != 728
    # one rounding of the output; fp16: of a subnormal
    bound = exact * 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -24
    assert (out[rest] - exact).abs().max() <= bound
