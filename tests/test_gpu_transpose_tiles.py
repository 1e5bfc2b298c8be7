"""The transpose's tiles: entries on both sides of a step of 32, of the eight steps read ahead, of a tile of
512 entries and of the size from which tiles hold 1,024, against a stable sort by column."""
import numpy as np
import pytest

from hsmu_gb import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nnz", [1, 31, 33, 255, 257, 511, 512, 513, 767, 3 * 512 + 256, (3 << 18) - 1, 3 << 18,
                                 (3 << 18) + 1, (3 << 18) + 1023, (3 << 18) + 1025])
def test_sizes(engine, nnz):
    import hsmu_gb

    rng = np.random.default_rng(nnz)
    M, N = 1 + nnz // 7, 70_000  # three digits
    per = np.full(M, nnz // M)
    per[: nnz % M] += 1
    rp = np.concatenate(([0], np.cumsum(per))).astype(np.int32)
    # increasing columns in every row: sorted distinct offsets from blocks of N / 16
    col = np.concatenate([np.sort(rng.choice(N, size=int(p), replace=False)) for p in per[:2000]]
                         + [(rng.integers(0, N // 16, size=int(p)) + (N // 16) * np.arange(int(p))) for p in per[2000:]])
    A = gen.CSR(M, N, rp, col.astype(np.int32), rng.uniform(-1, 1, nnz))
    T = engine.transpose(hsmu_gb.DeviceCSR.from_host(A)).to_host()
    row = np.repeat(np.arange(M), per)
    order = np.argsort(col, kind="stable")
    np.testing.assert_array_equal(T.row_ptr, np.concatenate(([0], np.cumsum(np.bincount(col.astype(int), minlength=N)))))
    np.testing.assert_array_equal(T.col, row[order])
    assert np.array_equal(T.val.view(np.int64), A.val[order].view(np.int64))
