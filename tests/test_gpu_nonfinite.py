"""Infinities and NaNs in A and B reach exactly the entries of C that their products belong to, on every path that
multiplies padding (steps that are not full, chains, networks, windows): bits equal the oracle's, NaN for NaN."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu


def spiked(A, seed):
    """a few infinities of both signs, NaNs, zeros and the largest and smallest values among A's"""
    rng = np.random.default_rng(seed)
    val = A.val.copy()
    special = np.array([np.inf, -np.inf, np.nan, 0.0, -0.0, np.finfo(float).max, -np.finfo(float).max, 5e-324])
    at = rng.choice(val.size, size=max(4, val.size // 400), replace=False)
    val[at] = special[rng.integers(0, special.size, at.size)]
    val[at[0]], val[at[1]] = np.inf, np.nan
    return gen.CSR(A.M, A.N, A.row_ptr, A.col, val)


def band(n, half):
    i = np.arange(n)[:, None]
    c = i + np.arange(-half, half + 1)[None, :]
    ok = (c >= 0) & (c < n)
    rp = np.concatenate(([0], np.cumsum(ok.sum(1)))).astype(np.int32)
    col = c[ok].astype(np.int32)
    return gen.CSR(n, n, rp, col, np.random.default_rng(half).uniform(-1, 1, col.size))


MATRICES = {
    "chains": lambda: gen.stencil27(8, 3),          # repeated rows
    "segments": lambda: gen.stencil27(12, 1),       # one segment after another
    "band": lambda: band(1500, 40),
    "tiny": lambda: gen.laplacian2d(40),            # networks
    "scattered": lambda: gen.poisson_random(60000, 6, seed=3),
    "windows": lambda: gen.rmat(12, 16, seed=5),    # windows, large rows
    "dense": lambda: band(300, 300),
}


def same(C, want):
    rp, col, val = want
    np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
    np.testing.assert_array_equal(C.col, col)
    nan = np.isnan(val)
    assert nan.any()
    np.testing.assert_array_equal(np.isnan(C.val), nan)
    assert np.array_equal(C.val[~nan].view(np.int64), val[~nan].view(np.int64))


@pytest.mark.parametrize("arith", [0, 1, 2])
@pytest.mark.parametrize("name", sorted(MATRICES))
def test_products(engine, name, arith):
    import torch

    import hsmu_gb
    from hsmu_gb import learned

    A = MATRICES[name]()
    A, B = spiked(A, 1), spiked(A, 2)
    dA, dB = hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)
    want = oracle.spgemm(A, B, fma=arith == 1)
    same(engine.spgemm(dA, dB, arith=arith).to_host(), want)
    same(engine.spgemm(dA, dB, arith=arith, tile_store=False).to_host(), want)
    params, margin, _ = learned.load()
    pt = torch.from_numpy(params).cuda()
    same(engine.spgemm_learned(dA, dB, pt, margin, arith=arith, always=True).to_host(), want)


@pytest.mark.parametrize("arith", [0, 1, 2])
def test_batches(engine, arith):
    # selecting tiles, short tiles, lists, rows for a warp and wide rows; A*P of a Galerkin product read again
    import hsmu_gb

    rng = np.random.default_rng(4)

    def rows(m, k, lo, hi):
        cols = [np.sort(rng.choice(k, n, replace=False)) for n in rng.integers(lo, hi + 1, m)]
        rp = np.concatenate(([0], np.cumsum([c.size for c in cols]))).astype(np.int32)
        return gen.CSR(m, k, rp, np.concatenate(cols).astype(np.int32), rng.uniform(-1, 1, int(rp[-1])))

    prods = [(rows(900, 300, 3, 8), rows(300, 60, 1, 1)), (rows(900, 300, 3, 8), rows(300, 60, 0, 4)),
             (gen.laplacian2d(25),) * 2, (gen.stencil27(6, 2),) * 2, (gen.rmat(10, 16, seed=3),) * 2]
    prods = [(spiked(a, 10 + i), spiked(b, 20 + i)) for i, (a, b) in enumerate(prods)]
    dev = lambda ms: [hsmu_gb.DeviceCSR.from_host(m) for m in ms]
    batch = hsmu_gb.Batch(engine, hsmu_gb.BATCH_PRODUCT, dev([a for a, _ in prods]), dev([b for _, b in prods]), arith=arith)
    batch.execute()
    batch.status()
    for p, (a, b) in enumerate(prods):
        same(batch.result(p).to_host(), oracle.spgemm(a, b, fma=arith == 1))
    batch.close()
    A = [spiked(gen.poisson7(9), 31), spiked(gen.poisson7(6), 32)]
    P = [gen.aggregation_prolongator(9), gen.aggregation_prolongator(6)]
    Pt = [gen.transpose(p) for p in P]
    batch = hsmu_gb.Batch(engine, hsmu_gb.BATCH_GALERKIN, dev(A), dev(P), dev(Pt), arith=arith)
    batch.execute()
    batch.status()
    for k in range(2):
        rp, col, val = oracle.spgemm(A[k], P[k], fma=arith == 1)
        AP = gen.CSR(A[k].M, P[k].N, rp.astype(np.int32), col, val)
        same(batch.result(k).to_host(), oracle.spgemm(Pt[k], AP, fma=arith == 1))
    batch.close()
