"""The value pass hands out the windows of long rows first, in the order of the rows: where every window is such
a one and B is several times the L2 cache, neighbouring windows still read the same rows of B together."""
import numpy as np
import pytest

from hsmu_gb import gen

pytestmark = pytest.mark.gpu


def windowed_products(A, side, dof):
    """products of the rows of A*A with more than 512 entries (27-point stencil: 5 nodes reached per axis)"""
    x = np.arange(side)
    reach = np.minimum(x, 2) + np.minimum(side - 1 - x, 2) + 1
    entries = dof * (reach[:, None, None] * reach[None, :, None] * reach[None, None, :]).ravel()
    per_row = np.add.reduceat(np.diff(A.row_ptr).astype(np.int64)[A.col], A.row_ptr[:-1])
    return int(per_row[np.repeat(entries, dof) > 512].sum())


def test_time_per_product_of_a_large_stencil(engine):
    # 27 points, 6 rows a node, rows of up to 162 entries: time per product on a grid whose B does not fit the
    # cache (300 MB) against one that does (37 MB)
    import hsmu_gb

    rate = []
    for side in (16, 30):
        A = gen.stencil27(side, 6)
        d = hsmu_gb.DeviceCSR.from_host(A)
        ms = []
        for _ in range(8):
            engine.spgemm(d, d, stats=True).free()
            ms.append(engine.last_stats["ms_numeric"])
        rate.append(min(ms) / windowed_products(A, side, 6))
    # 0.98 in order, 1.14 in any order
    assert rate[1] < 1.06 * rate[0], (rate, rate[1] / rate[0])
