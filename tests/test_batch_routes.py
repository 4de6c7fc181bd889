"""Which sets of 1D problems a batch advances in the resident kernel (one launch for many stages) and which in stage
launches: the faster of the two for the set, with the same bits."""
import numpy as np
import pytest

from test_flat2d import kinds, wave

pytestmark = pytest.mark.gpu
STAGES = 32
# (problems, cells of each): measured, resident / stage launches, in us per stage
SETS = {
    (160, 124): "resident",  # 3.7 / 7.6
    (2400, 124): "resident",  # 17.4 / 21.4
    (75, 1000): "resident",  # 5.7 / 8.3
    (9, 4096): "resident",  # 5.5 / 7.9
    (150, 1000): "stages",  # 12.9 / 10.4
    (48, 4096): "stages",  # 20.4 / 16.6
    (50, 6000): "stages",  # 40.3 / 17.3
    (9, 8192): "stages",  # 12.7 / 8.0
}


@pytest.mark.parametrize("count,n", sorted(SETS))
def test_long_runs(count, n, tslib):
    from turbostructred_gb300 import capi
    case = capi.make_case(ndims=1, nx=n, periodic=(0, 1, 1), recon=3, solver=1, cfl=0.4, max_iter=10 ** 6, max_time=1e30,
                          bc=kinds("natural"))
    ic, res = wave(n, 1, 1), []
    for tail in (True, False):
        with capi.Batch(1 << 30) as b:
            b.set_tail(tail)
            ids = [b.add(case, ic) for _ in range(count)]
            b.step(STAGES)
            launches = b.stats()["launches"]
            res.append([b.get(i) for i in ids[:: max(1, count // 4)]])
        assert launches == 1 if tail and SETS[count, n] == "resident" else launches >= STAGES
    for (u, a), (v, c) in zip(*res):
        assert np.array_equal(u, v) and a["time"] == c["time"] and a["iteration"] == c["iteration"] == STAGES
