"""Selecting tiles of the batched engine: left rows around the limit of eight entries, right rows with
no, one and two entries (the last send the rest of the product to the insertion lists), products that
change kind from one to the next, partial tiles, every arithmetic, against the oracle."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu


def rows_of(lengths, k, seed):
    rng = np.random.default_rng(seed)
    cols = [np.sort(rng.choice(k, size=min(int(n), k), replace=False)) for n in lengths]
    rp = np.concatenate(([0], np.cumsum([c.size for c in cols]))).astype(np.int32)
    col = np.concatenate(cols).astype(np.int32) if rp[-1] else np.zeros(0, np.int32)
    return gen.CSR(len(lengths), k, rp, col, rng.uniform(-1, 1, col.size))


def selector(k, n, seed, empty=0.0, two=()):
    rng = np.random.default_rng(seed)
    lens = np.where(rng.random(k) < empty, 0, 1)
    for i in two:
        lens[i] = 2
    return rows_of(lens, n, seed + 1)


def products():
    rng = np.random.default_rng(5)
    out = []
    # rows of 0..8 entries, few right columns (runs of up to eight equal ones) and many
    for M, n in ((1, 1), (31, 3), (32, 5), (33, 400), (1000, 7), (3001, 2000)):
        out.append((rows_of(rng.integers(0, 9, M), 300, M), selector(300, n, M + 50, empty=0.2)))
    # a row of nine entries in some tile; a right row of two entries met late; a plain product between
    lens = np.full(500, 7)
    lens[321] = 9
    out.append((rows_of(lens, 200, 7), selector(200, 40, 8)))
    out.append((rows_of(np.full(700, 6), 900, 9), selector(900, 50, 10, two=(899,))))
    out.append((gen.laplacian2d(20, seed=1), gen.laplacian2d(20, seed=2)))
    out.append((rows_of(np.full(257, 8), 64, 11), selector(64, 64, 12)))
    return out


@pytest.mark.parametrize("grid", [0, 1])  # every tile to another warp; all tiles of a warp's in turn
@pytest.mark.parametrize("arith", [0, 1, 2])
def test_selecting_products(engine, arith, grid):
    import hsmu_gb

    prods = products()
    A = [hsmu_gb.DeviceCSR.from_host(a) for a, _ in prods]
    B = [hsmu_gb.DeviceCSR.from_host(b) for _, b in prods]
    batch = hsmu_gb.Batch(engine, hsmu_gb.BATCH_PRODUCT, A, B, arith=arith)
    for tiny in (32, 8, 7):
        batch.set_params(tiny, grid)
        batch.execute()
        batch.status()
        for p, (a, b) in enumerate(prods):
            C = batch.result(p).to_host()
            rp, col, val = oracle.spgemm(a, b, fma=arith == 1)
            np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
            np.testing.assert_array_equal(C.col, col)
            assert np.array_equal(C.val.view(np.int64), val.view(np.int64)), (tiny, p)
    batch.close()


def test_negative_zero_and_cancellation(engine):
    # a lone product -0.0 becomes 0.0 + -0.0 = 0.0; products that cancel leave their entry
    import hsmu_gb

    A = gen.CSR(2, 4, np.array([0, 1, 4], np.int32), np.array([0, 1, 2, 3], np.int32), np.array([-0.0, 1.0, -1.0, 2.0]))
    B = gen.CSR(4, 3, np.array([0, 1, 2, 3, 4], np.int32), np.array([2, 1, 1, 0], np.int32), np.ones(4))
    batch = hsmu_gb.Batch(engine, hsmu_gb.BATCH_PRODUCT, [hsmu_gb.DeviceCSR.from_host(A)],
                          [hsmu_gb.DeviceCSR.from_host(B)])
    batch.execute()
    batch.status()
    C = batch.result(0).to_host()
    rp, col, val = oracle.spgemm(A, B)
    np.testing.assert_array_equal(C.col, col)
    assert np.array_equal(C.val.view(np.int64), val.view(np.int64))
    batch.close()


def test_selecting_tiles_in_turn(engine):
    # more tiles than the launch has warps, so that a warp meets tiles ahead of it: within a product, across
    # a product that cannot have selecting tiles, and after a tile that is not one
    import hsmu_gb

    lens = np.full(200_001, 7)
    lens[[40_000, 199_999]] = 9
    prods = [(rows_of(np.arange(130_000) % 9, 500, 20), selector(500, 80, 21, empty=0.1)),
             (gen.laplacian2d(30, seed=3), gen.laplacian2d(30, seed=4)),
             (rows_of(lens, 300, 22), selector(300, 90, 23)),
             (rows_of(np.full(120_000, 8), 64, 24), selector(64, 50, 25, two=(63,)))]
    prods[3] = (prods[3][0], gen.CSR(64, 50, *trim(prods[3][1])))
    batch = hsmu_gb.Batch(engine, hsmu_gb.BATCH_PRODUCT, [hsmu_gb.DeviceCSR.from_host(a) for a, _ in prods],
                          [hsmu_gb.DeviceCSR.from_host(b) for _, b in prods])
    for _ in range(2):
        batch.execute()
        batch.status()
        for p, (a, b) in enumerate(prods):
            C = batch.result(p).to_host()
            rp, col, val = oracle.spgemm(a, b)
            np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
            np.testing.assert_array_equal(C.col, col)
            assert np.array_equal(C.val.view(np.int64), val.view(np.int64)), p
    batch.close()


def test_last_column_of_the_widest_keys(engine):
    # column 2^27 - 1 as the 32nd product of a row: its sort key must not be the empty one
    import hsmu_gb

    n = 1 << 27
    col = np.tile(np.array([0, 1, 2, 3]), 8)
    col[-1] = n - 1
    A = gen.CSR(1, 8, np.array([0, 8], np.int32), np.arange(8, dtype=np.int32), np.arange(1.0, 9.0))
    B = gen.CSR(8, n, np.arange(0, 33, 4, dtype=np.int32), col.astype(np.int32), np.ones(32))
    batch = hsmu_gb.Batch(engine, hsmu_gb.BATCH_PRODUCT, [hsmu_gb.DeviceCSR.from_host(A)],
                          [hsmu_gb.DeviceCSR.from_host(B)])
    batch.execute()
    batch.status()
    C = batch.result(0).to_host()
    np.testing.assert_array_equal(C.col, [0, 1, 2, 3, n - 1])
    np.testing.assert_array_equal(C.val, [36.0, 36.0, 36.0, 28.0, 8.0])
    batch.close()


def trim(b):
    """b without its first entry: row 63 keeps two, and there are no more entries than rows."""
    rp = np.maximum(np.asarray(b.row_ptr) - 1, 0).astype(np.int32)
    return rp, b.col[1:], b.val[1:]


def short_products():
    rng = np.random.default_rng(15)
    out = []
    # rows of 0..8 entries against rows of 0..4: few columns (long runs) and many
    for M, n in ((1, 1), (31, 4), (32, 6), (33, 5000), (2000, 9), (1501, 300)):
        out.append((rows_of(rng.integers(0, 9, M), 250, M), rows_of(rng.integers(0, 5, 250), n, M + 70)))
    out.append((rows_of(np.full(400, 8), 100, 16), rows_of(np.full(100, 4), 7, 17)))  # 32 products, 7 columns
    out.append((rows_of(np.full(400, 8), 100, 18), rows_of(np.full(100, 4), 4000, 19)))  # 32 products, mostly distinct
    lens = np.full(300, 4)
    lens[257] = 5  # a right row of five entries met late: the lists from there
    out.append((rows_of(np.full(900, 5), 300, 20), rows_of(lens, 60, 21)))
    lens = np.full(500, 8)
    lens[340] = 9
    out.append((rows_of(lens, 200, 22), rows_of(np.full(200, 3), 90, 23)))
    return out


@pytest.mark.parametrize("grid", [0, 1])
@pytest.mark.parametrize("arith", [0, 1, 2])
def test_short_products(engine, arith, grid):
    import hsmu_gb

    prods = short_products()
    A = [hsmu_gb.DeviceCSR.from_host(a) for a, _ in prods]
    B = [hsmu_gb.DeviceCSR.from_host(b) for _, b in prods]
    batch = hsmu_gb.Batch(engine, hsmu_gb.BATCH_PRODUCT, A, B, arith=arith)
    for tiny in (32, 31):
        batch.set_params(tiny, grid)
        batch.execute()
        batch.status()
        for p, (a, b) in enumerate(prods):
            C = batch.result(p).to_host()
            rp, col, val = oracle.spgemm(a, b, fma=arith == 1)
            np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
            np.testing.assert_array_equal(C.col, col)
            assert np.array_equal(C.val.view(np.int64), val.view(np.int64)), (tiny, p)
    batch.close()


def test_short_second_product(engine):
    # Galerkin batches whose second product is short for some grids and not for others
    import hsmu_gb

    sides = [16, 5, 9, 33, 2, 1]
    A, P, Pt = [], [], []
    for k, s in enumerate(sides):
        A.append(gen.poisson7(s, seed=k))
        p = gen.aggregation_prolongator(s)
        if k == 2:  # aggregates of random size: rows of P^T beyond eight entries
            rng = np.random.default_rng(3)
            p = gen.CSR(p.M, 11, p.row_ptr, rng.integers(0, 11, p.M).astype(np.int32), p.val)
        P.append(p)
        Pt.append(gen.transpose(p))
    dev = lambda ms: [hsmu_gb.DeviceCSR.from_host(m) for m in ms]
    batch = hsmu_gb.Batch(engine, hsmu_gb.BATCH_GALERKIN, dev(A), dev(P), dev(Pt))
    batch.execute()
    batch.status()
    for p in range(len(sides)):
        rp, col, val = oracle.spgemm(A[p], P[p])
        AP = gen.CSR(A[p].M, P[p].N, rp.astype(np.int32), col, val)
        rp, col, val = oracle.spgemm(Pt[p], AP)
        C = batch.result(p).to_host()
        np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
        np.testing.assert_array_equal(C.col, col)
        assert np.array_equal(C.val.view(np.int64), val.view(np.int64)), p
    batch.close()
