"""Tiny rows with one entry of A, whose row of C is a row of B: warps of only such rows, warps with a longer row
among them, empty rows and rows of B, values whose sums with 0.0 matter, against the oracle."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu


def csr(rows, n, vals):
    rp = np.concatenate(([0], np.cumsum([len(r) for r in rows]))).astype(np.int32)
    col = np.concatenate([np.asarray(r, np.int32) for r in rows]).astype(np.int32)
    return gen.CSR(len(rows), n, rp, col, vals(int(rp[-1])))


@pytest.mark.parametrize("arith", [0, 1, 2])
@pytest.mark.parametrize("longer", [0, 1, 40])  # rows of two entries per thousand
def test_rows_of_one_entry(engine, arith, longer):
    import torch

    import hsmu_gb
    from hsmu_gb import learned

    rng = np.random.default_rng(longer)
    # B rows of 0, 1, 7, 8, 9, 15, 16, 17, 31 and 32 entries (and 33: the next class)
    lens = [0, 1, 7, 8, 9, 15, 16, 17, 31, 32, 33] * 5
    vals = lambda n: np.where(rng.random(n) < 0.2, -0.0, rng.uniform(-1, 1, n))
    B = csr([np.sort(rng.choice(3000, k, replace=False)) for k in lens], 3000, vals)
    short = [k for k, n in enumerate(lens) if n <= 9]
    rows = []
    for i in range(3001):
        if i % 1000 < longer:
            rows.append(np.sort(rng.choice(short, 2, replace=False)))
        else:
            rows.append([] if i % 11 == 5 else [rng.integers(0, len(lens))])
    A = csr(rows, len(lens), vals)
    dA, dB = hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)
    rp, col, val = oracle.spgemm(A, B, fma=arith == 1)
    params, margin, _ = learned.load()
    pt = torch.from_numpy(params).cuda()
    for C in (engine.spgemm(dA, dB, arith=arith), engine.spgemm_learned(dA, dB, pt, margin, arith=arith, always=True)):
        C = C.to_host()
        np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
        np.testing.assert_array_equal(C.col, col)
        assert np.array_equal(C.val.view(np.int64), val.view(np.int64))
    np.testing.assert_array_equal(engine.row_nnz(dA, dB).cpu().numpy(), np.diff(rp))


def test_gathered_rows_are_not_sorted(engine):
    # three million rows that each take a row of 27, alone and with a second entry of A whose B row is empty (such
    # rows are listed and sorted): 1,141 and 1,505 us in the fill kernel
    import hsmu_gb

    rng = np.random.default_rng(5)
    M, K, b = 3_000_000, 2000, 27
    cols = np.sort(rng.integers(0, 3000, (K, b)), axis=1) + np.arange(b)
    brp = np.minimum(np.arange(K + 2) * b, K * b).astype(np.int32)
    B = gen.CSR(K + 1, 5000, brp, cols.astype(np.int32).ravel(), rng.uniform(-1, 1, K * b))
    dB = hsmu_gb.DeviceCSR.from_host(B)
    pick = rng.integers(0, K, M).astype(np.int32)
    best = []
    for k in (1, 2):
        col = np.stack([pick, np.full(M, K, np.int32)], axis=1)[:, :k]
        A = gen.CSR(M, K + 1, np.arange(0, M * k + 1, k, dtype=np.int32), col.ravel(), rng.uniform(-1, 1, M * k))
        dA = hsmu_gb.DeviceCSR.from_host(A)
        ms = []
        for _ in range(8):
            engine.spgemm(dA, dB, stats=True).free()
            ms.append(engine.last_stats["ms_structure"])
        best.append(min(ms))
    assert best[0] < 0.88 * best[1], best
