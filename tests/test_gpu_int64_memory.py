"""hsmu_spgemm64 where the windows of all rows together are more than its limit for one symbolic pass, or more
than the memory that is left: the panels are then run one by one, and the product is the same."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu

HSMU_ERR_ALLOC = 2
GIB = 1 << 30


def free_bytes():
    import torch

    return torch.cuda.mem_get_info()[0]


# one-entry rows of A over rows of 33 columns from the first to the last of 2^31 - 1: a large row has a window
# bound of 8,192, whatever its entries.  30,000 rows: 11.8 GB of windows, more than the limit; 8,000 rows: 3.1 GB
@pytest.mark.parametrize("rows,left_gib", [(30000, 6), (8000, 2)])
def test_windows_beyond_the_limit_or_the_memory(rows, left_gib):
    import gc

    import torch

    import hsmu_gb

    rng = np.random.default_rng(7)
    N = (1 << 31) - 1
    K, n = 5, 33
    cols = np.sort(rng.integers(1, N - 1, size=(K, n)).astype(np.int64), axis=1)
    cols[:, 0], cols[:, -1] = 0, N - 1
    assert (np.diff(cols, axis=1) > 0).all()
    B = gen.CSR(K, N, np.arange(0, K * n + 1, n, dtype=np.int32), cols.astype(np.int32).ravel(), rng.uniform(-1, 1, K * n))
    pick = rng.integers(0, K, rows).astype(np.int32)
    A = gen.CSR(rows, K, np.arange(rows + 1, dtype=np.int32), pick, rng.uniform(-1, 1, rows))
    dA, dB = hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)
    eng = hsmu_gb.Engine()
    warm = gen.laplacian2d(8)
    eng.spgemm(hsmu_gb.DeviceCSR.from_host(warm), hsmu_gb.DeviceCSR.from_host(warm)).free()
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(max(0, free_bytes() - left_gib * GIB), dtype=torch.uint8, device="cuda")
    try:
        C = eng.spgemm64(dA, dB, max_panel_nnz=33 * 1000)
        rp, col, val = C.to_host()
        C.free()
    finally:
        del hog
        torch.cuda.empty_cache()
        eng.close()
    np.testing.assert_array_equal(rp, np.arange(0, rows * n + 1, n))
    np.testing.assert_array_equal(col.reshape(rows, n), cols[pick])
    want = 0.0 + A.val[:, None] * B.val.reshape(K, n)[pick]
    assert np.array_equal(val.reshape(rows, n).view(np.int64), want.view(np.int64))


def test_failures_while_the_pass_takes_memory(engine):
    # every allocation in turn fails once: the call reports it or, past the point where the panels can be run
    # one by one, finishes
    import hsmu_gb

    A = gen.rmat(12, 16, seed=3)
    dA = hsmu_gb.DeviceCSR.from_host(A)
    want = oracle.spgemm(A, A)
    reported = 0
    for nth in range(1, 80):
        hsmu_gb.debug_fail_alloc(nth)
        try:
            C = engine.spgemm64(dA, dA, max_panel_nnz=40000)
        except hsmu_gb.HsmuError as e:
            assert e.status == HSMU_ERR_ALLOC, (nth, e)
            reported += 1
            continue
        finally:
            hsmu_gb.debug_fail_alloc(0)
        rp, col, val = C.to_host()
        C.free()
        np.testing.assert_array_equal(rp, want[0])
        np.testing.assert_array_equal(col, want[1])
        assert np.array_equal(val.view(np.int64), want[2].view(np.int64))
    assert 3 <= reported < 79
