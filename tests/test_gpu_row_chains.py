"""Chains of B rows with one pattern (k_row_repeat, the chain path of hsmu_products.cuh): every run
length around the chain limit, leaders of many lengths, neighbouring chains that share columns, and
A rows that enter a run anywhere, bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu


def repeated_rows(runs, ncols, lo, hi, seed):
    """B: groups of `runs[g % len(runs)]` rows with one random pattern each (lo..hi columns)"""
    rng = np.random.default_rng(seed)
    rp, cols = [0], []
    g = 0
    while len(rp) < 800:
        c = np.sort(rng.choice(ncols, size=rng.integers(lo, hi + 1), replace=False))
        for _ in range(runs[g % len(runs)]):
            cols.append(c)
            rp.append(rp[-1] + c.size)
        g += 1
    col = np.concatenate(cols).astype(np.int32)
    return gen.CSR(len(rp) - 1, ncols, np.array(rp, np.int32), col, rng.uniform(-1, 1, col.size))


def windows_of_rows(m, k, width, seed):
    """A: each row references a run of consecutive B rows with a few left out"""
    rng = np.random.default_rng(seed)
    rp, cols = [0], []
    for i in range(m):
        s = int(rng.integers(0, k))
        c = np.arange(s, min(k, s + width))
        c = c[rng.random(c.size) < (1.0 if i % 2 else 0.9)]
        cols.append(c)
        rp.append(rp[-1] + c.size)
    col = np.concatenate(cols).astype(np.int32)
    return gen.CSR(m, k, np.array(rp, np.int32), col, rng.uniform(-1, 1, col.size))


CASES = {
    # runs of 1..7 rows (chains of 3, remainders 1 and 2), leaders of 36..100 columns
    "runs1to7": ((1, 2, 3, 4, 5, 6, 7), 300, 36, 100, 90),
    # narrow matrix: successive chains share most of their columns (the two-round adds)
    "overlap": ((2, 3), 110, 60, 100, 70),
    # a full column block (every slot taken), one row per step boundary: 32, 64, 96 columns
    "full": ((3,), 96, 96, 96, 64),
    # leaders too short for chains (the other paths), with repeats
    "short": ((3, 4), 400, 8, 30, 120),
    # leaders on both sides of the limit
    "mixed": ((3, 1, 6), 480, 2, 120, 50),
}


@pytest.mark.parametrize("arith", [0, 1, 2])
@pytest.mark.parametrize("name", sorted(CASES))
def test_repeated_rows(engine, name, arith):
    import hsmu_gb

    runs, ncols, lo, hi, width = CASES[name]
    B = repeated_rows(runs, ncols, lo, hi, seed=3)
    A = windows_of_rows(300, B.M, width, seed=4)
    C = engine.spgemm(hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B), arith=arith).to_host()
    rp, col, val = oracle.spgemm(A, B, fma=arith == 1)
    np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
    np.testing.assert_array_equal(C.col, col)
    assert np.array_equal(C.val.view(np.int64), val.view(np.int64))


@pytest.mark.parametrize("dof", [2, 3, 4, 6])
def test_stencil_blocks(engine, dof):
    import hsmu_gb

    A = gen.stencil27(7, dof, seed=dof)
    dA = hsmu_gb.DeviceCSR.from_host(A)
    C = engine.spgemm(dA, dA).to_host()
    C2 = engine.spgemm(dA, dA, tiles=hsmu_gb.BTiles(engine, dA)).to_host()
    rp, col, val = oracle.spgemm(A, A)
    for X in (C, C2):
        np.testing.assert_array_equal(X.row_ptr.astype(np.int64), rp)
        np.testing.assert_array_equal(X.col, col)
        assert np.array_equal(X.val.view(np.int64), val.view(np.int64))


@pytest.mark.parametrize("run", [1, 2, 3, 4, 5, 8, 31, 32, 33, 40])
def test_repeated_rows_of_a(engine, run):
    # A's rows repeat in runs around the group of four and the 32 rows a run's place is told from; B is
    # another matrix, with rows long enough to look for repeats, and outputs with and without windows
    import hsmu_gb

    rng = np.random.default_rng(run)
    base = [np.sort(rng.choice(500, size=int(rng.integers(36, 60)), replace=False)) for _ in range(200 // run + 2)]
    cols = [c for c in base for _ in range(run)]
    rp = np.concatenate(([0], np.cumsum([c.size for c in cols]))).astype(np.int32)
    col = np.concatenate(cols).astype(np.int32)
    A = gen.CSR(len(cols), 500, rp, col, rng.uniform(-1, 1, col.size))
    for ncols in (300, 9000):
        B = repeated_rows((1, 3), ncols, 40, 60, seed=run)
        B = gen.CSR(500, ncols, B.row_ptr[:501], B.col[:B.row_ptr[500]], B.val[:B.row_ptr[500]])
        dA, dB = hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)
        want = oracle.spgemm(A, B)
        np.testing.assert_array_equal(engine.row_nnz(dA, dB).cpu().numpy(), np.diff(want[0]))
        C = engine.spgemm(dA, dB).to_host()
        rp64, col64, val64 = engine.spgemm64(dA, dB, max_panel_nnz=5000).to_host()
        np.testing.assert_array_equal(C.row_ptr.astype(np.int64), want[0])
        np.testing.assert_array_equal(rp64, want[0])
        for c, v in ((C.col, C.val), (col64, val64)):
            np.testing.assert_array_equal(c, want[1])
            assert np.array_equal(v.view(np.int64), want[2].view(np.int64))
