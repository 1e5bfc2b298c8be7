"""Rows of many entries: both sides of the length from which the bounds and feature passes take a row
with a block (256), of the products from which a narrow row leaves the warp class (24,576), and B rows
around the steps of the tile pass (multiples of 32 and 128), against the oracle."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu


def rows_of(lengths, k, seed):
    rng = np.random.default_rng(seed)
    cols = [np.sort(rng.choice(k, size=n, replace=False)) for n in lengths]
    rp = np.concatenate(([0], np.cumsum(lengths))).astype(np.int32)
    return gen.CSR(len(lengths), k, rp, np.concatenate(cols).astype(np.int32), rng.uniform(-1, 1, int(rp[-1])))


def operands(span):
    # B rows of 128 columns: 192 entries of A are 24,576 products, 193 are 24,704
    lengths = [255, 256, 257, 192, 193, 1, 0, 700, 1900, 300, 31, 2] * 20 + [256, 257]
    A = rows_of(lengths, 2000, seed=1)
    B = rows_of([128] * 2000, span, seed=2)
    assert A.nnz >= 1 << 16 and A.nnz > 6 * A.M
    return A, B


def same(C, want):
    rp, col, val = want
    np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
    np.testing.assert_array_equal(C.col, col)
    assert np.array_equal(C.val.view(np.int64), val.view(np.int64))


@pytest.mark.parametrize("span", [3000, 30000, 50000])
def test_long_rows(engine, span):
    import torch

    import hsmu_gb
    from hsmu_gb import learned

    A, B = operands(span)
    dA, dB = hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)
    want = oracle.spgemm(A, B)
    for store in (True, True, False):
        same(engine.spgemm(dA, dB, tile_store=store).to_host(), want)
    params, margin, _ = learned.load()
    pt = torch.from_numpy(params).cuda()
    same(engine.spgemm_learned(dA, dB, pt, margin, always=True).to_host(), want)
    nnz = engine.row_nnz(dA, dB).cpu().numpy()
    np.testing.assert_array_equal(nnz, np.diff(want[0]))


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 1000])
def test_tiles_of_row_lengths(engine, n):
    import hsmu_gb

    B = rows_of([n, 0, n, max(1, n - 1), n + 1] * 8, 40 * n + 70, seed=n)
    got = hsmu_gb.BTiles(engine, hsmu_gb.DeviceCSR.from_host(B)).arrays()
    rows = np.repeat(np.arange(B.M), np.diff(B.row_ptr))
    t = (B.col >> 6).astype(np.int64)
    first = np.ones(B.nnz, bool)
    first[1:] = (t[1:] != t[:-1]) | (rows[1:] != rows[:-1])
    starts = np.flatnonzero(first)
    ptr = np.zeros(B.M + 1, np.int64)
    np.cumsum(np.bincount(rows[starts], minlength=B.M), out=ptr[1:])
    mask = np.bitwise_or.reduceat(np.left_shift(np.uint64(1), (B.col & 63).astype(np.uint64)), starts)
    for g, w in zip(got, (ptr, t[starts], mask, starts)):
        np.testing.assert_array_equal(g.astype(np.uint64), w.astype(np.uint64))
