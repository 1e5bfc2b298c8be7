"""Two handles in two threads at once, each with its own stream: scratch, side stream and scan state belong to the
handle, and the pools that the handles share are the driver's."""
import threading

import numpy as np
import pytest

import oracle
from hsmu_gb import gen

pytestmark = pytest.mark.gpu


def test_two_handles_in_two_threads():
    import torch

    import hsmu_gb

    mats = [gen.rmat(13, 16, seed=6), gen.poisson_random(40000, 12, seed=7), gen.stencil27(14, 3), gen.laplacian2d(150)]
    want = [oracle.spgemm(m, m) for m in mats]
    dev = [hsmu_gb.DeviceCSR.from_host(m) for m in mats]
    batches_in = [gen.laplacian2d(20 + k) for k in range(6)]
    batch_want = [oracle.spgemm(m, m) for m in batches_in]
    batch_dev = [hsmu_gb.DeviceCSR.from_host(m) for m in batches_in]
    torch.cuda.synchronize()
    errors = []
    start = threading.Barrier(2)

    def same(C, w):
        assert np.array_equal(C.row_ptr.astype(np.int64), w[0])
        assert np.array_equal(C.col, w[1])
        assert np.array_equal(C.val.view(np.int64), w[2].view(np.int64))

    def work(t):
        try:
            st = torch.cuda.Stream()
            eng = hsmu_gb.Engine()
            start.wait(30)
            for k in range(24):
                i = (k + t * 2 + k // 5) % len(mats)
                C = eng.spgemm(dev[i], dev[i], stream=st)
                same(C.to_host(stream=st), want[i])
                C.free()
                if k % 6 == t:
                    rp, col, val = eng.spgemm64(dev[i], dev[i], max_panel_nnz=200000, stream=st).to_host(stream=st)
                    same(gen.CSR(mats[i].M, mats[i].N, rp, col, val), want[i])
                if k % 6 == 3:
                    r = eng.spgemm_host(mats[i], mats[i], stream=st)
                    same(gen.CSR(mats[i].M, mats[i].N, *r), want[i])
                if k % 8 == 4:
                    b = hsmu_gb.Batch(eng, hsmu_gb.BATCH_PRODUCT, batch_dev, batch_dev, stream=st)
                    b.execute(stream=st)
                    b.status(stream=st)
                    for p, w in enumerate(batch_want):
                        same(b.result(p).to_host(stream=st), w)
                    b.close()
            eng.close()
        except BaseException as e:  # shown by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors, errors
    assert not any(t.is_alive() for t in threads)
