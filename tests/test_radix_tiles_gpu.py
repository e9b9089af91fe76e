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


@pytest.mark.parametrize("n, room", [(909311, 909312), (3000, 3000), (908000, 908000)])
def test_workspaces_of_large_tiles_are_taken(n, room):
    """The size without the longer table of small tiles: 12 bytes a key, 1024 for each 2048 keys, the scan's and 64."""
    from sparseswin3d_b200 import _lib

    tiles = -(-room // 2048)
    k = torch.randint(-2 ** 31, 2 ** 31, (n,), generator=torch.Generator().manual_seed(n)).to(torch.int32)
    size = 12 * room + 1024 * tiles + 8 * (2 + -(-256 * tiles // 2048)) + 64
    keys, out = k.cuda(), torch.empty(n, dtype=torch.int32, device="cuda")
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    args = keys.data_ptr(), n, out.data_ptr(), ws.data_ptr()
    assert _lib.lib.ssw_argsort_i32(*args, size - 4 * (room - n) * 3 - 8192, _lib.stream_ptr(out.device)) == -5   # (nothing is launched)
    assert _lib.lib.ssw_argsort_i32(*args, size, _lib.stream_ptr(out.device)) == 0
    assert torch.equal(out.cpu(), O.sort_indices(k))
