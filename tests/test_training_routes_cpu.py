"""From how many rows a Linear that trains goes through the library's own passes, without a GPU."""
import pytest
import torch


@pytest.mark.parametrize("rows_, narrow, dtype, few", [
    (16383, 96, torch.float32, True), (16384, 96, torch.float32, False), (16384, 48, torch.float32, False), (16383, 48, torch.float32, True),
    (4999, 192, torch.float32, True), (5000, 192, torch.float32, False), (2499, 384, torch.float32, True), (2500, 384, torch.float32, False),
    (2499, 767, torch.float32, True), (1023, 768, torch.float32, True), (1024, 768, torch.float32, False), (1023, 3072, torch.float32, True),
    (99999, 96, torch.bfloat16, True), (100000, 96, torch.bfloat16, False), (50000, 192, torch.float16, False)])
def test_rows_from_which_the_passes_pay(rows_, narrow, dtype, few):
    from sparseswin3d_b200 import rows

    assert rows._few_for_training(rows_, narrow, dtype) == few


@pytest.mark.parametrize("narrow", [96, 192, 384, 768, 1536])
@pytest.mark.parametrize("wide", [1, 3, 4])
def test_products_of_the_backward_pay_where_the_passes_do(narrow, wide):
    from sparseswin3d_b200 import rows

    m = next(m for m in range(1, 20000) if not rows._few_for_training(m, narrow, torch.float32))
    for n, k in ((narrow, wide * narrow), (wide * narrow, narrow)):
        assert rows._gemm_pays(m, n, k)
