"""A new handle is ready when hsmu_handle_create returns: its first calls, on a stream that does not wait for the
default one, are right while the default stream still has earlier work queued."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu


def test_first_calls_beside_work_queued_on_the_default_stream():
    import torch

    import hsmu_gb

    A = gen.poisson_random(40000, 12, seed=1)  # scans and binning over several tiles
    want = oracle.spgemm(A, A)
    dA = hsmu_gb.DeviceCSR.from_host(A)
    side = torch.cuda.Stream()
    x = torch.randn(4096, 4096, device="cuda")
    torch.matmul(x, x)
    torch.cuda.synchronize()
    for _ in range(3):
        for _ in range(40):  # some tens of milliseconds
            y = torch.matmul(x, x)
        eng = hsmu_gb.Engine()
        results = [eng.spgemm(dA, dA, stream=side) for _ in range(3)]
        torch.cuda.synchronize()
        for C in results:
            got = C.to_host()
            np.testing.assert_array_equal(got.row_ptr.astype(np.int64), want[0])
            np.testing.assert_array_equal(got.col, want[1])
            assert np.array_equal(got.val.view(np.int64), want[2].view(np.int64))
            C.free()
        eng.close()
        del y
