"""Backward of the fused attention at the edges of its tiles, against float64 autograd of the dense restatement."""
import pytest
import torch

from oracle import ssw_oracle as O
from tests.cases import rel_err

pytestmark = pytest.mark.gpu

# largest error over the result's size: fp32 sums of up to 1000 terms, fp16 / bf16 one rounding of the row gradients
# (2^-11, 2^-8 at values near the rms; smaller values are measured against the rms)
TOL = {torch.float32: 3e-5, torch.float16: 1.5e-3, torch.bfloat16: 1.2e-2}


def _windows(counts, w, seed):
    """One window per entry of `counts`, that many voxels in it, listed in random order."""
    g = torch.Generator().manual_seed(seed)
    rows = []
    for k, c in enumerate(counts):
        pos = torch.randperm(w ** 3, generator=g)[:c]
        rows.append(torch.stack([torch.zeros_like(pos), k * w + pos // (w * w), pos // w % w, pos % w], 1))
    coords = torch.cat(rows).int()
    return coords[torch.randperm(len(coords), generator=g)].contiguous(), (len(counts) * w, w, w)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("counts,w,heads,hd", [
    ([1, 2, 3, 1], 7, 3, 32),                          # less than a pack
    ([31, 32, 33, 63, 64, 1, 16, 17] * 2, 7, 3, 32),   # half and whole tiles
    ([65, 127, 128, 129, 343, 5], 7, 2, 16),           # windows beyond a pack: remainders of key and query tiles
    ([1000, 64, 200], 10, 2, 32),                      # table too large for the shared-memory columns
    ([40, 70, 12], 7, 12, 32),                         # wide rows: smaller tiles in the plan
])
def test_backward_at_tile_edges(dtype, counts, w, heads, hd):
    from sparseswin3d_b200 import attention, window

    coords, dims = _windows(counts, w, seed=sum(counts))
    n, scale = len(coords), hd ** -0.5
    g = torch.Generator().manual_seed(n)
    qkv = torch.randn(n, 3, heads, hd, generator=g).to(dtype)
    go = torch.randn(n, heads * hd, generator=g).to(dtype)
    table = torch.randn((2 * w - 1) ** 3, heads, generator=g) * 0.5
    geom = window.resolve_geometry(1, dims, (w,) * 3)
    plan = window.bucket_windows(coords=coords.cuda(), geom=geom, **attention.plan_params(heads, hd, dtype, (w,) * 3))
    dq, dt = attention.window_attention_fused_backward(qkv.cuda(), go.cuda(), plan, table.cuda(), scale)
    plan.raise_on_error()
    q64, t64 = qkv.double().requires_grad_(True), table.double().requires_grad_(True)
    idx = O.window_keys(coords, 1, dims, (w,) * 3, (0, 0, 0))[0]
    out = O.dense_window_attention(q64, idx, scale, t64, O.relative_position_index((w,) * 3))
    rq, rt = torch.autograd.grad(out.reshape(n, -1), (q64, t64), go.double())
    assert rel_err(dq.double().cpu(), rq) <= TOL[dtype]
    assert rel_err(dt.double().cpu(), rt) <= 1e-4      # fp32 whatever the rows' type
