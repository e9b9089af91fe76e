"""The radix sort around the edges of its tiles (1024 and 2048 keys) and of its warps' runs, with digits that fill a tile alone."""
import pytest
import torch

from oracle import ssw_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1023, 1024, 1025, 8191, 444 * 2048 - 1, 444 * 2048, 444 * 2048 + 2049])
@pytest.mark.parametrize("keys", ["equal", "two", "signed", "descending"])
def test_stable_order(n, keys):
    from sparseswin3d_b200 import ops

    g = torch.Generator().manual_seed(n)
    k = {"equal": torch.full((n,), -7),
         "two": torch.randint(0, 2, (n,), generator=g) * 0x01010101 - 1,
         "signed": torch.randint(-2 ** 31, 2 ** 31, (n,), generator=g),
         "descending": -torch.arange(n)}[keys].to(torch.int32)
    assert torch.equal(ops.sort_indices(k.cuda()).cpu(), O.sort_indices(k))
