"""GEMMs of different sums from several threads: a launch must not be refused for the shared memory that another caller's took."""
import sys
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_gemms_of_several_threads():
    from sparseswin3d_b200._lib import lib

    results = []

    def work(k):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            x, w = torch.randn(300, k, device="cuda"), torch.randn(96, k, device="cuda")
            out = torch.empty(300, 96, device="cuda")
            args = x.data_ptr(), w.data_ptr(), 0, out.data_ptr(), 300, 96, k, 0, stream.cuda_stream
            refused = sum(lib.ssw_gemm_f32(*args) != 0 for _ in range(10000))
            ref = x.double() @ w.double().t()
            # 24 bits of the operands, sums of 192 terms at most: an ulp of the result, by its norm
            results.append((refused, float((out - ref).norm() / ref.norm()) < 2e-7))

    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-5)
    try:
        threads = [threading.Thread(target=work, args=(k,)) for k in (192, 32, 192, 32)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    assert results == [(0, True)] * 4
