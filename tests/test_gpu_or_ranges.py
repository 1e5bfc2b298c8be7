"""The large rows' OR walk with long B rows apart (warp_or_tiles, LONG): ranges of 127, 128 and 129 tiles,
one unit of four steps and its neighbours, among short and empty ones; rows inside one chunk of the tile
table and across several; more and fewer long ranges than warps, against the oracle."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu

TILES = (0, 1, 3, 31, 33, 127, 128, 129, 160, 255, 256, 257, 513)


def build(span, seed):
    rng = np.random.default_rng(seed)
    rows = []
    for i in range(13 * 20):
        t = np.sort(rng.choice(span, size=TILES[i % 13], replace=False))
        rows.append(np.unique(np.concatenate([t * 64 + rng.integers(0, 64, t.size) for _ in range(1 + i % 2)])
                              if t.size else t))
    rp = np.concatenate(([0], np.cumsum([r.size for r in rows]))).astype(np.int32)
    B = gen.CSR(len(rows), span * 64, rp, np.concatenate(rows).astype(np.int32), rng.uniform(-1, 1, rp[-1]))
    arows = []
    for kinds in ((5,), (6,), (7,), (1, 2, 3, 6), (6, 7, 12), (0, 1, 5), (8, 9, 10, 11, 12), tuple(range(13))):
        for n in (33, 40, 64, 70, 150):
            pool = np.flatnonzero(np.isin(np.arange(260) % 13, kinds))
            arows.append(np.sort(rng.choice(260, size=min(n, 260), replace=False)) if len(kinds) == 13
                         else np.union1d(rng.choice(pool, size=min(n, pool.size), replace=False),
                                         rng.choice(np.arange(2, 260, 13), size=18, replace=False)))
    arp = np.concatenate(([0], np.cumsum([r.size for r in arows]))).astype(np.int32)
    A = gen.CSR(len(arows), 260, arp, np.concatenate(arows).astype(np.int32), rng.uniform(-1, 1, arp[-1]))
    return A, B


@pytest.mark.parametrize("span", [520, 4096, 4097, 9000])
def test_ranges(engine, span):
    import hsmu_gb

    A, B = build(span, span)
    dA, dB = hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)
    rp, col, val = oracle.spgemm(A, B)
    for store in (True, False):
        C = engine.spgemm(dA, dB, validate=True, tile_store=store).to_host()
        np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
        np.testing.assert_array_equal(C.col, col)
        assert np.array_equal(C.val.view(np.int64), val.view(np.int64))
