"""The value pass's hand-out of windows (k_numeric): rows on both sides of the lengths from which
their windows are listed first, alone and mixed, in one call and in row panels, against the oracle."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu


def rows_of(lengths, k, seed):
    rng = np.random.default_rng(seed)
    cols = [np.sort(rng.choice(k, size=n, replace=False)) for n in lengths]
    rp = np.concatenate(([0], np.cumsum(lengths))).astype(np.int32)
    col = np.concatenate(cols).astype(np.int32) if len(cols) else np.zeros(0, np.int32)
    return gen.CSR(len(lengths), k, rp, col, rng.uniform(-1, 1, col.size))


CASES = {
    "edges": [127, 128, 129, 511, 512, 513, 40, 0, 900],
    "listed_only": [600] * 5 + [200] * 5,
    "unlisted_only": [100, 127, 64] * 4,
    "one_heavy_last": [90] * 20 + [1500],
}


@pytest.mark.parametrize("span", [30000, 90000])  # warp-class rows; large rows with tile lists
@pytest.mark.parametrize("name", sorted(CASES))
def test_window_order(engine, name, span):
    import hsmu_gb

    A = rows_of(CASES[name], 2000, seed=1)
    B = gen.poisson_random(2000, 25, seed=2, ncols=span)
    dA, dB = hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)
    rp, col, val = oracle.spgemm(A, B)
    for _ in range(2):  # the second call has the tile store's arena
        C = engine.spgemm(dA, dB, stats=True)
        assert engine.last_stats["windows"] > 0
        C = C.to_host()
        np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
        np.testing.assert_array_equal(C.col, col)
        assert np.array_equal(C.val.view(np.int64), val.view(np.int64))
    p_rp, p_col, p_val = engine.spgemm64(dA, dB, max_panel_nnz=6000).to_host()
    np.testing.assert_array_equal(p_rp, rp)
    np.testing.assert_array_equal(p_col, col)
    assert np.array_equal(p_val.view(np.int64), val.view(np.int64))
