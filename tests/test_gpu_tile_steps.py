"""B's tile conversion: rows on both sides of one step of 32 entries, tiles that end with a step or run through
several, the kept tiles against a plain restatement; rows of one step cost no more than their share."""
import numpy as np
import pytest

from hsmu_gb import gen

pytestmark = pytest.mark.gpu


def tiles_of(B):
    ptr, tcol, mask, off = [0], [], [], []
    for k in range(B.M):
        s, e = int(B.row_ptr[k]), int(B.row_ptr[k + 1])
        c = B.col[s:e].astype(np.int64)
        t, first = np.unique(c >> 6, return_index=True)
        for i, f in enumerate(first):
            last = first[i + 1] if i + 1 < len(first) else e - s
            tcol.append(t[i])
            mask.append(np.bitwise_or.reduce(np.uint64(1) << (c[f:last] & 63).astype(np.uint64)))
            off.append(s + f)
        ptr.append(len(tcol))
    return np.array(ptr), np.array(tcol), np.array(mask, dtype=np.uint64), np.array(off)


def test_tiles_of_short_and_long_rows(engine):
    import hsmu_gb

    rng = np.random.default_rng(1)
    lens = [0, 1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 161, 400] * 6
    rows = []
    for i, n in enumerate(lens):
        span = (n + 1, 64 * 3 + n, 5000)[i // 18 % 3]  # dense, a few per tile, mostly one per tile
        rows.append(np.sort(rng.choice(span, n, replace=False)) + int(rng.integers(0, 200)))
    rp = np.concatenate(([0], np.cumsum(lens))).astype(np.int32)
    B = gen.CSR(len(lens), 6000, rp, np.concatenate(rows).astype(np.int32), rng.uniform(-1, 1, int(rp[-1])))
    t = hsmu_gb.BTiles(engine, hsmu_gb.DeviceCSR.from_host(B))
    for got, want in zip(t.arrays(), tiles_of(B)):
        np.testing.assert_array_equal(got, want)
    t.free()


@pytest.mark.parametrize("n", [1, 20, 32])
@pytest.mark.parametrize("what", ["order", "twice", "range"])
def test_rows_of_one_step_are_checked(engine, n, what):
    # validation of the conversion's input (the kernels read no more than the row)
    import hsmu_gb

    if n == 1 and what != "range":
        pytest.skip("one entry has no neighbour")
    col = np.arange(0, 3 * n, 3, dtype=np.int32)
    if what == "order":
        col[[0, 1]] = col[[1, 0]]
    elif what == "twice":
        col[1] = col[0]
    else:
        col[-1] = 500
    B = gen.CSR(2, 500, np.array([0, n, n], np.int32), col, np.ones(n))
    with pytest.raises(hsmu_gb.HsmuError) as ei:
        hsmu_gb.BTiles(engine, hsmu_gb.DeviceCSR.from_host(B))
    assert ei.value.status == 5  # HSMU_ERR_UNSORTED


def test_conversion_of_short_rows(engine):
    # a million rows of eight and of nine entries: nine cost no more than nine eighths (rows of nine took a loop of
    # four steps before)
    import torch

    import hsmu_gb

    rng = np.random.default_rng(2)
    best = []
    for n in (8, 9):
        m = 1_000_000
        col = np.sort(rng.integers(0, 60000, (m, n)), axis=1) + np.arange(n)
        B = gen.CSR(m, 60100, np.arange(0, m * n + 1, n, dtype=np.int32), col.astype(np.int32).ravel(), np.ones(m * n))
        d = hsmu_gb.DeviceCSR.from_host(B)
        times = []
        for _ in range(10):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            t = hsmu_gb.BTiles(engine, d)
            t1.record()
            torch.cuda.synchronize()
            times.append(t0.elapsed_time(t1))
            t.free()
        best.append(min(times))
    assert best[1] < 9 / 8 * best[0], best
