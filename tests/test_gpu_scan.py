"""Single-pass scans and binning (k_rows.cu): row counts on both sides of a tile, of the number of tiles
looked back over at once, and of the most tiles of a launch (4,096), where a tile takes several pieces.
Rows of A hold one entry each, so C's row pointers and entries follow from B's rows."""
import numpy as np
import pytest

from hsmu_gb import gen

pytestmark = pytest.mark.gpu


def operands(M, seed):
    """A: one entry per row (every 7th row none), B: rows of 0, 1, 20, 200 and 900 columns: tiny rows,
    warp rows with and without windows, scattered and large rows"""
    rng = np.random.default_rng(seed)
    big = M <= 100000
    lens = [0, 1, 3, 20] + ([200, 900, 300] if big else [])
    span = [1, 40, 5000, 60000] + ([30000, 30000, 90000] if big else [])
    N = 90000
    rows = [np.sort(rng.choice(s, size=n, replace=False)) for n, s in zip(lens, span)]
    rp = np.concatenate(([0], np.cumsum(lens))).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    B = gen.CSR(len(lens), N, rp, col, rng.uniform(-1, 1, col.size))
    pick = rng.integers(0, len(lens), size=M).astype(np.int32)
    if big and M > 3000:  # few long rows
        rare = rng.random(M) > 0.02
        pick[rare] = pick[rare] % 4
    has = np.arange(M) % 7 != 3
    arp = np.concatenate(([0], np.cumsum(has))).astype(np.int32)
    A = gen.CSR(M, len(lens), arp, pick[has], rng.uniform(-1, 1, int(arp[-1])))
    return A, B


@pytest.mark.parametrize("M", [1, 31, 1023, 1024, 1025, 2047, 2048, 2049, 33 * 1024 + 5, 33 * 2048 + 7, 4096 * 1024 + 3,
                               4096 * 2048 + 9])
def test_row_counts(engine, M):
    import hsmu_gb

    A, B = operands(M, seed=M % 1000)
    dA, dB = hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)
    C = engine.spgemm(dA, dB).to_host()
    n = np.zeros(M, np.int64)
    has = np.diff(A.row_ptr) > 0
    blen = np.diff(B.row_ptr)
    n[has] = blen[A.col]
    rp = np.concatenate(([0], np.cumsum(n)))
    np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
    # entry e of C is entry e - rp[row] of the B row that the row references
    at = np.repeat(B.row_ptr[A.col].astype(np.int64), n[has]) + (np.arange(rp[-1]) - np.repeat(rp[:-1][has], n[has]))
    np.testing.assert_array_equal(C.col, B.col[at])
    val = np.repeat(A.val, n[has]) * B.val[at]
    assert np.array_equal(C.val.view(np.int64), (0.0 + val).view(np.int64))
    rp64, col64, val64 = engine.spgemm64(dA, dB, max_panel_nnz=max(1, int(rp[-1]) // 3)).to_host()
    np.testing.assert_array_equal(rp64, rp)
    np.testing.assert_array_equal(col64, C.col)
    assert np.array_equal(val64.view(np.int64), C.val.view(np.int64))


def test_many_calls_on_two_streams(engine):
    # the look-back words are told apart by their launch, not cleared: every call's scans find only
    # their own, whichever stream the call runs on
    import torch

    import hsmu_gb

    side = torch.cuda.Stream()
    cases = []
    for M in (5000, 40000, 2049):
        A, B = operands(M, seed=M)
        cases.append((hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)))
    want = [engine.spgemm(a, b).to_host() for a, b in cases]
    torch.cuda.synchronize()
    for k in range(60):
        a, b = cases[k % 3]
        C = engine.spgemm(a, b, stream=side if k % 2 else None).to_host()
        np.testing.assert_array_equal(C.row_ptr, want[k % 3].row_ptr)
        np.testing.assert_array_equal(C.col, want[k % 3].col)
