"""Which tiles of a batch take which way: rows of one entry keep the insertion lists (a row of B is in order
already), and the selecting tiles' launch is left out where too few tiles could be selecting ones."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu


def rows_of(lengths, k, seed):
    rng = np.random.default_rng(seed)
    cols = [np.sort(rng.choice(k, size=int(n), replace=False)) for n in lengths]
    rp = np.concatenate(([0], np.cumsum([c.size for c in cols]))).astype(np.int32)
    return gen.CSR(len(lengths), k, rp, np.concatenate(cols).astype(np.int32), rng.uniform(-1, 1, int(rp[-1])))


def fixed_rows(m, k, n, seed):
    rng = np.random.default_rng(seed)
    col = np.sort(rng.integers(0, n - k, (m, k)), axis=1) + np.arange(k)
    return gen.CSR(m, n, np.arange(0, m * k + 1, k, dtype=np.int32), col.astype(np.int32).ravel(), rng.uniform(-1, 1, m * k))


def batch_of(engine, prods, **kw):
    import hsmu_gb

    return hsmu_gb.Batch(engine, hsmu_gb.BATCH_PRODUCT, [hsmu_gb.DeviceCSR.from_host(a) for a, _ in prods],
                         [hsmu_gb.DeviceCSR.from_host(b) for _, b in prods], **kw)


def check(batch, prods, arith):
    batch.status()
    for p, (a, b) in enumerate(prods):
        C = batch.result(p).to_host()
        rp, col, val = oracle.spgemm(a, b, fma=arith == 1)
        np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
        np.testing.assert_array_equal(C.col, col)
        assert np.array_equal(C.val.view(np.int64), val.view(np.int64)), p


@pytest.mark.parametrize("arith", [0, 1, 2])
def test_rows_of_one_entry(engine, arith):
    rng = np.random.default_rng(1)
    prods = [(rows_of(rng.integers(0, 2, 1000), 300, 2), rows_of(rng.integers(0, 5, 300), 90, 3)),
             # tiles of one-entry rows, then tiles with longer ones, then one-entry rows again
             (rows_of(np.concatenate((np.ones(200), rng.integers(2, 9, 200), np.ones(200))), 250, 4),
              rows_of(rng.integers(0, 5, 250), 40, 5))]
    batch = batch_of(engine, prods, arith=arith)
    batch.execute()
    check(batch, prods, arith)
    batch.close()


def kernels_of(fn):
    import torch
    from torch.profiler import ProfilerActivity, profile

    for _ in range(2):  # the process's first session may see no kernels
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            fn()
            torch.cuda.synchronize()
    return [e.name for e in prof.events() if "k_batch" in e.name]


# 5,000 rows, 157 tiles; rows of nine entries (not selecting): none, as many as half of the tiles, one more
@pytest.mark.parametrize("nine,selects", [(0, True), (78, True), (79, False), (2500, False)])
def test_selecting_launch(engine, nine, selects):
    lens = np.full(5000, 6)
    lens[np.random.default_rng(3).choice(5000, nine, replace=False)] = 9
    prods = [(rows_of(lens, 700, 6), rows_of(np.ones(700), 200, 7))]
    batch = batch_of(engine, prods)
    names = kernels_of(batch.execute)
    check(batch, prods, 0)
    assert any("k_batch_select" in n for n in names) == selects, names
    assert len(names) == 1 + selects, names
    batch.close()


def test_gathered_rows_of_four(engine):
    # 200,000 rows that each take a row of four or of five entries, integer products: five cost more than four
    # (four took the network of 32, and its 32 products, before)
    import torch

    best = []
    for k in (4, 5):
        prods = [(fixed_rows(200000, 1, 500, i), fixed_rows(500, k, 3000, i + 9)) for i in range(4)]
        batch = batch_of(engine, prods, arith=2)
        times = []
        for _ in range(10):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            batch.execute()
            t1.record()
            torch.cuda.synchronize()
            times.append(t0.elapsed_time(t1))
        best.append(min(times))
        batch.close()
    assert best[0] < best[1], best
