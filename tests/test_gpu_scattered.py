"""Scattered rows (k_scatter.cu): both sides of every limit of the class -- products (32/33, 512/513),
A entries (32/33), tile span (512/513, 16384/16385) -- rows with and without repeated columns, empty
B rows in between, every arithmetic, and the learned path's slots, bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu


def csr(rows, ncols, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate(([0], np.cumsum([len(r) for r in rows]))).astype(np.int32)
    col = np.concatenate([np.sort(np.asarray(r, np.int64)) for r in rows]).astype(np.int32)
    return gen.CSR(len(rows), ncols, rp, col, rng.uniform(-1, 1, col.size))


def rows_with(products, entries, pool, rng):
    """`entries` B rows (indices into pool) whose lengths add up to `products`"""
    lens = np.full(entries, products // entries)
    lens[:products % entries] += 1
    used = {}
    out = []
    for n in lens:
        k = used.get(int(n), 0)
        used[int(n)] = k + 1
        out.append(pool[int(n)][k])
    return out


def build(span_tiles, ncols_extra, dense, seed):
    """A, B: rows of A on both sides of the product and entry limits; B rows of every length used,
    each holding the first and last column of the span; dense: few distinct columns, so rows repeat
    them"""
    rng = np.random.default_rng(seed)
    first, last = 64 * 3 + 5, 64 * 3 + 64 * (span_tiles - 1) + 60
    ncols = last + 1 + ncols_extra
    wants = [(33, 3), (32, 2), (64, 4), (511, 16), (512, 16), (513, 16), (200, 32), (200, 33), (512, 32), (512, 31),
             (40, 1), (500, 1), (512, 1), (513, 1)]
    lens = set()
    for p, e in wants:
        lens.add(p // e)
        lens.add(p // e + 1)
    pool, rows = {}, [[] for _ in range(5)]  # a few empty B rows first
    inner = np.unique(rng.integers(first + 1, last, size=700 if dense else 200000))
    for n in sorted(lens):
        pool[n] = []
        for _ in range(34):
            mid = rng.choice(inner, size=max(0, n - 2), replace=False)
            pool[n].append(len(rows))
            rows.append(np.concatenate(([first], mid, [last]))[:n] if n >= 2 else [first if _ % 2 else last])
    B = csr(rows, ncols, seed + 1)
    A = csr([rows_with(p, e, pool, rng) + [0, 3][:int(e < 31)] for p, e in wants], B.M, seed + 2)
    return A, B


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("span", [512, 513, 3000, 16384, 16385])
@pytest.mark.parametrize("arith", [0, 1, 2])
def test_limits(engine, span, dense, arith):
    import hsmu_gb

    A, B = build(span, 100, dense, seed=span)
    C = engine.spgemm(hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B), arith=arith, validate=True)
    C = C.to_host()
    rp, col, val = oracle.spgemm(A, B, fma=arith == 1)
    np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
    np.testing.assert_array_equal(C.col, col)
    assert np.array_equal(C.val.view(np.int64), val.view(np.int64))


@pytest.mark.parametrize("margin", [0.8, -40.0])  # slots that fit, slots that all overflow
def test_learned_slots(engine, margin):
    import torch

    import hsmu_gb
    from hsmu_gb import learned

    A, B = build(3000, 0, True, seed=9)
    dA, dB = hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)
    params = torch.from_numpy(learned.load()[0]).cuda()
    C = engine.spgemm_learned(dA, dB, params, margin, always=True, stats=True)
    assert engine.last_stats["routed"] == 0
    if margin < 0:
        assert engine.last_stats["fallback_rows"] > 0
    C = C.to_host()
    rp, col, val = oracle.spgemm(A, B)
    np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
    np.testing.assert_array_equal(C.col, col)
    assert np.array_equal(C.val.view(np.int64), val.view(np.int64))


def test_uniform_rows(engine):
    # most rows without a repeated column, some with, tiny and large rows among them
    import hsmu_gb

    A = gen.poisson_random(40001, 7, seed=3)
    dA = hsmu_gb.DeviceCSR.from_host(A)
    C = engine.spgemm(dA, dA).to_host()
    rp, col, val = oracle.spgemm(A, A)
    np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
    np.testing.assert_array_equal(C.col, col)
    assert np.array_equal(C.val.view(np.int64), val.view(np.int64))
