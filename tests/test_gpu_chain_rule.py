"""The chain kernel (repeated B rows) is launched only where B's rows form few chains: shares of chains on both
sides of the line, bit for bit against the oracle; and rows without repeats are no slower for being long enough
to be looked at."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu


def runs(n_rows, run, single, ncols, seed):
    """rows in runs of `run` equal patterns, after each of which `single` rows stand alone; 40..70 columns"""
    rng = np.random.default_rng(seed)
    cols = []
    while len(cols) < n_rows:
        c = np.sort(rng.choice(ncols, size=rng.integers(40, 71), replace=False))
        cols += [c] * run
        cols += [np.sort(rng.choice(ncols, size=rng.integers(40, 71), replace=False)) for _ in range(single)]
    cols = cols[:n_rows]
    rp = np.concatenate(([0], np.cumsum([c.size for c in cols]))).astype(np.int32)
    return gen.CSR(n_rows, ncols, rp, np.concatenate(cols).astype(np.int32), rng.uniform(-1, 1, int(rp[-1])))


# (rows of a run, single rows after it): 33, 41, 44, 47, 50, 60 and 100 % of the rows start a chain
@pytest.mark.parametrize("run,single", [(3, 0), (15, 2), (9, 3), (12, 3), (6, 2), (2, 0), (3, 2), (1, 0)])
@pytest.mark.parametrize("always", [False, True])  # the plain call, the predicted slots
def test_shares_around_the_line(engine, run, single, always):
    import torch

    import hsmu_gb
    from hsmu_gb import learned

    B = runs(700, run, single, 480, seed=run * 10 + single)
    rng = np.random.default_rng(run)
    acols = [np.arange(s, min(700, s + int(w))) for s, w in zip(rng.integers(0, 690, 400), rng.integers(1, 50, 400))]
    arp = np.concatenate(([0], np.cumsum([c.size for c in acols]))).astype(np.int32)
    A = gen.CSR(400, 700, arp, np.concatenate(acols).astype(np.int32), rng.uniform(-1, 1, int(arp[-1])))
    dA, dB = hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)
    if always:
        params, margin, _ = learned.load()
        C = engine.spgemm_learned(dA, dB, torch.from_numpy(params).cuda(), margin, always=True).to_host()
    else:
        C = engine.spgemm(dA, dB).to_host()
    rp, col, val = oracle.spgemm(A, B)
    np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
    np.testing.assert_array_equal(C.col, col)
    assert np.array_equal(C.val.view(np.int64), val.view(np.int64))


def band(n, half):
    i = np.arange(n)[:, None]
    c = i + np.arange(-half, half + 1)[None, :]
    ok = (c >= 0) & (c < n)
    rp = np.concatenate(([0], np.cumsum(ok.sum(1)))).astype(np.int32)
    col = c[ok].astype(np.int32)
    return gen.CSR(n, n, rp, col, np.random.default_rng(half).uniform(-1, 1, col.size))


def test_bands_without_repeated_rows(engine):
    # 33 entries a row: too short to be looked at; 61: looked at, none repeats.  The wider band has 3.4 times the
    # products and fills its steps of 32 better, so its time per product is about half (1.24 times the narrow
    # one's where the chain kernel is launched for it)
    import torch

    import hsmu_gb

    per_product = []
    for half in (16, 30):
        A = band(40000, half)
        d = hsmu_gb.DeviceCSR.from_host(A)
        times = []
        for _ in range(8):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            C = engine.spgemm(d, d)
            t1.record()
            torch.cuda.synchronize()
            times.append(t0.elapsed_time(t1))
            C.free()
        per_product.append(min(times) / gen.products(A, A))
    assert per_product[1] < 0.85 * per_product[0], per_product
