"""The single-launch scans wait for earlier blocks' sums, for a bounded number of polls (hsmu_opts.scan_polls, a
test hook).  A scan that gives up leaves bins, row pointers, tile pointers or window positions unfinished: no
kernel of the call may index by them, the call reports HSMU_ERR_TIMEOUT, and the next one on the handle is right."""
import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu

HSMU_ERR_TIMEOUT = 7


def operands(seed):
    """40,000 rows of every class: tiny, warp rows with and without windows, scattered, large; B of 6,000 rows"""
    rng = np.random.default_rng(seed)
    K, N = 6000, 70000
    lens = rng.choice([0, 1, 3, 20, 60, 300], size=K, p=[.05, .4, .3, .15, .08, .02])
    span = rng.choice([2000, 20000, N], size=K)
    cols = [np.sort(rng.choice(s, size=n, replace=False)) for n, s in zip(lens, span)]
    rp = np.concatenate(([0], np.cumsum(lens))).astype(np.int32)
    B = gen.CSR(K, N, rp, np.concatenate(cols).astype(np.int32), rng.uniform(-1, 1, int(rp[-1])))
    M = 40000
    alen = rng.choice([0, 1, 5, 14, 200], size=M, p=[.05, .4, .4, .1495, .0005])
    acol = [np.sort(rng.choice(K, size=n, replace=False)) for n in alen]
    arp = np.concatenate(([0], np.cumsum(alen))).astype(np.int32)
    A = gen.CSR(M, K, arp, np.concatenate(acol).astype(np.int32), rng.uniform(-1, 1, int(arp[-1])))
    return A, B


def calls(engine, A, B, dA, dB):
    import torch

    from hsmu_gb import learned

    params, margin, _ = learned.load()
    pt = torch.from_numpy(params).cuda()

    def wide(C):
        rp, col, val = C.to_host()
        return gen.CSR(A.M, B.N, rp.astype(np.int32), col, val)

    return {
        "plain": lambda: engine.spgemm(dA, dB).to_host(),
        "no store": lambda: engine.spgemm(dA, dB, tile_store=False).to_host(),
        "learned": lambda: engine.spgemm_learned(dA, dB, pt, margin, always=True).to_host(),
        "int64": lambda: wide(engine.spgemm64(dA, dB, max_panel_nnz=900000)),
        "host": lambda: gen.CSR(A.M, B.N, *engine.spgemm_host(A, B)),
    }


def test_scans_that_give_up(engine, monkeypatch):
    import hsmu_gb

    A, B = operands(3)
    dA, dB = hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)
    rp, col, val = oracle.spgemm(A, B)
    plain_opts = hsmu_gb.c_opts

    def hurried(*a):
        o = plain_opts(*a)
        o.scan_polls = 1
        return o

    def exact(C):
        np.testing.assert_array_equal(C.row_ptr.astype(np.int64), rp)
        np.testing.assert_array_equal(C.col, col)
        assert np.array_equal(C.val.view(np.int64), val.view(np.int64))

    for name, call in calls(engine, A, B, dA, dB).items():
        gave_up = 0
        for _ in range(12):
            monkeypatch.setattr(hsmu_gb, "c_opts", hurried)
            try:
                exact(call())  # every sum was there at the first poll
            except hsmu_gb.HsmuError as e:
                assert e.status == HSMU_ERR_TIMEOUT, (name, e)
                gave_up += 1
            monkeypatch.setattr(hsmu_gb, "c_opts", plain_opts)
            exact(call())
        assert gave_up > 0, name
