"""Tiny rows (at most 32 products, a thread each, sorted by a network in registers): warps whose longest
row has 0, 1, 8, 9, 16, 17, 31 and 32 products, rows of another class beside them, empty B rows in
between, repeated and distinct columns, row panels, every arithmetic, and the widest column counts that a
sort key holds, bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu

LENGTHS = (0, 1, 2, 3, 5, 8, 32, 33)


def build(ncols, distinct, seed):
    """B: rows of LENGTHS[i % 8] entries (few columns, or all over with the last one always in);
    A: 64 rows per product limit, made of B rows that add up to at most the limit"""
    rng = np.random.default_rng(seed)
    rows = []
    for i in range(160):
        n = LENGTHS[i % 8]
        c = set(rng.integers(0, ncols if distinct else 40, size=4 * n + 8).tolist())
        c = set(rng.permutation(sorted(c))[:max(0, n - 1)].tolist()) | {ncols - 1} if n else set()
        while len(c) < n:
            c.add(int(rng.integers(0, min(ncols, 400))))
        rows.append(sorted(c))
    rp = np.concatenate(([0], np.cumsum([len(r) for r in rows]))).astype(np.int32)
    B = gen.CSR(160, ncols, rp, np.concatenate(rows).astype(np.int32), rng.uniform(-1, 1, rp[-1]))
    arows = []
    for limit in (0, 1, 8, 9, 16, 17, 31, 32, 33):
        for i in range(64):
            left, take = limit if i % 3 else int(rng.integers(0, limit + 1)), set()
            for k in rng.permutation(160):
                if LENGTHS[k % 8] <= left:
                    take.add(int(k))
                    left -= LENGTHS[k % 8]
            arows.append(sorted(take))
    arp = np.concatenate(([0], np.cumsum([len(r) for r in arows]))).astype(np.int32)
    A = gen.CSR(len(arows), 160, arp, np.concatenate(arows).astype(np.int32), rng.uniform(-1, 1, arp[-1]))
    return A, B


@pytest.mark.parametrize("distinct", [False, True])
@pytest.mark.parametrize("ncols", [64, 5000, (1 << 27) - 1, (1 << 27) + 3])
def test_tiny_rows(engine, ncols, distinct):
    import hsmu_gb

    A, B = build(ncols, distinct, 3)
    dA, dB = hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)
    for arith in (0, 1, 2):
        C = engine.spgemm(dA, dB, arith=arith).to_host()
        rp, col, val = reference(A, B, arith)
        np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
        np.testing.assert_array_equal(C.col, col)
        assert np.array_equal(C.val.view(np.int64), val.view(np.int64)), arith


def reference(A, B, arith):
    # columns renumbered to those that B holds: the oracle's work arrays are as long as a row
    used, inv = np.unique(B.col, return_inverse=True)
    small = gen.CSR(B.M, used.size, B.row_ptr, inv.astype(np.int32), B.val)
    rp, col, val = oracle.spgemm(A, small, fma=arith == 1)
    return rp, used[col], val
