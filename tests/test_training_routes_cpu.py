"""From how many rows a Linear that trains goes through the library's own passes, without a GPU."""
import pytest
import torch


@pytest.mark.parametrize("rows_, narrow, dtype, few", [
    (16383, 96, torch.float32, True), (16384, 96, torch.float32, False), (16384, 48, torch.float32, False), (16383, 48, torch.float32, True),
    (4095, 192, torch.float32, True), (4096, 192, torch.float32, False), (1023, 384, torch.float32, True), (1024, 384, torch.float32, False),
    (99999, 96, torch.bfloat16, True), (100000, 96, torch.bfloat16, False), (50000, 192, torch.float16, False)])
def test_rows_from_which_the_passes_pay(rows_, narrow, dtype, few):
    from sparseswin3d_b200 import rows

    assert rows._few_for_training(rows_, narrow, dtype) == few
