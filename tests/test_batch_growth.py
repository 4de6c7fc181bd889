"""Batches whose tables of descriptors and control words grow (from 64 problems on) while others run and finish."""
import numpy as np
import pytest

from test_flat2d import kinds, wave

pytestmark = pytest.mark.gpu


def problem(k):
    from turbostructred_gb300 import capi
    n = 16 + 3 * (k % 11)
    return capi.make_case(ndims=1, nx=n, periodic=(k % 2, 1, 1), recon=3 * (k % 3 > 0), solver=1 + 2 * (k % 2), cfl=0.4,
                          max_iter=5 + k % 7, max_time=1e30, bc=kinds("symmetry")), (1.0 + 0.01 * (k % 5)) * wave(n, 1, 1)


def alone(k):
    from turbostructred_gb300 import capi
    with capi.Batch(16 << 20) as b:
        i = b.add(*problem(k))
        b.run()
        return b.get(i)


@pytest.mark.parametrize("count", [63, 64, 65, 129, 300])
@pytest.mark.parametrize("tail", [True, False])
def test_problems_added_one_by_one(count, tail, tslib):
    """A problem whose addition made the tables grow, and those around it: as each alone."""
    from turbostructred_gb300 import capi
    with capi.Batch(64 << 20) as b:
        b.set_tail(tail)
        ids = []
        for k in range(count):
            ids.append(b.add(*problem(k)))
            if k % 16 == 15:
                b.step(2)  # some are under way, and from the second time on some have ended
            if k in (64, 128):
                got = b.get(ids[0])  # read on the download stream right after the growth
                want = alone(0)
                assert np.array_equal(got[0], want[0]) and got[1]["iteration"] == 5
        b.run()
        got = [b.get(i) for i in ids]
    want = {}
    for k, (u, info) in enumerate(got):
        key = (k % 11, k % 2, k % 3 > 0, k % 7, k % 5)
        if key not in want:
            want[key] = alone(k)
        v, ref = want[key]
        assert np.array_equal(u, v) and info["time"] == ref["time"] and info["iteration"] == ref["iteration"]
