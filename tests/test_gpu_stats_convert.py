"""hsmu_stats.ms_convert is the time of B's tile conversion, whatever its place in the call: with a small B
under many rows of A it is a small part of the symbolic time, which holds the bounds pass over A's rows."""
import numpy as np
import pytest

from hsmu_gb import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [2, 40])  # tiny rows (their tiles are read by no row), warp rows
def test_conversion_of_a_small_right_operand(engine, lens):
    import hsmu_gb

    rng = np.random.default_rng(1)
    K, M = 64, 6_000_000
    B = gen.CSR(K, 4096, np.arange(0, K * lens + 1, lens, dtype=np.int32),
                np.concatenate([np.sort(rng.choice(4096, lens, replace=False)) for _ in range(K)]).astype(np.int32),
                rng.uniform(-1, 1, K * lens))
    A = gen.CSR(M, K, np.arange(M + 1, dtype=np.int32), rng.integers(0, K, M).astype(np.int32), rng.uniform(-1, 1, M))
    dA, dB = hsmu_gb.DeviceCSR.from_host(A), hsmu_gb.DeviceCSR.from_host(B)
    share = []
    for _ in range(6):
        C = engine.spgemm(dA, dB, stats=True)
        C.free()
        s = engine.last_stats
        share.append(s["ms_convert"] / s["ms_symbolic"])
        assert s["ms_total"] >= s["ms_convert"] + s["ms_symbolic"]
    assert min(share) < 0.2, share
