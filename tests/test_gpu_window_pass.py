"""The window length pass where a block takes several pieces of the windows (more than 4,194,304 of them): rows
whose windows are listed first among rows whose are not, against the oracle on renumbered columns."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [500, 530, 1100])  # window bound 8,192 a row: one, two and three pieces
def test_pieces(engine, rows):
    import hsmu_gb

    rng = np.random.default_rng(rows)
    N = (1 << 31) - 1
    K, n = 700, 40
    cols = np.sort(rng.integers(1, N - 1, size=(K, n)).astype(np.int64), axis=1)
    cols[:, 0], cols[:, -1] = 0, N - 1
    cols[:, 20] = cols[0, 20] if cols[:, 19].max() < cols[0, 20] < cols[:, 21].min() else cols[:, 20]
    assert (np.diff(cols, axis=1) > 0).all()
    B = gen.CSR(K, N, np.arange(0, K * n + 1, n, dtype=np.int32), cols.astype(np.int32).ravel(), rng.uniform(-1, 1, K * n))
    lens = np.ones(rows, int)
    at = rng.choice(rows, 24, replace=False)
    lens[at] = [127, 128, 129, 130] * 4 + [511, 512, 513, 600] * 2
    acol = [np.sort(rng.choice(K, k, replace=False)) for k in lens]
    A = gen.CSR(rows, K, np.concatenate(([0], np.cumsum(lens))).astype(np.int32), np.concatenate(acol).astype(np.int32),
                rng.uniform(-1, 1, int(lens.sum())))
    dA, dB = hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)
    ids = np.unique(cols)
    small = gen.CSR(K, ids.size, B.row_ptr, np.searchsorted(ids, cols).astype(np.int32).ravel(), B.val)
    rp, col, val = oracle.spgemm(A, small)
    for store in (True, True, False):
        C = engine.spgemm(dA, dB, tile_store=store).to_host()
        np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
        np.testing.assert_array_equal(C.col, ids[col])
        assert np.array_equal(C.val.view(np.int64), val.view(np.int64))
