"""1D problems of two and three cells (the fewest that are accepted) on the mixed path: in the resident kernel, alone
and among others in a batch, with the stage kernels' bits."""
import numpy as np
import pytest

from test_flat2d import SIDES, kinds, wave

pytestmark = pytest.mark.gpu


def case(n, k, **kw):
    from turbostructred_gb300 import capi
    bc = sorted(SIDES)[k % len(SIDES)]
    return capi.make_case(ndims=1, nx=n, periodic=(k % 2, 1, 1), recon=(0, 1, 2, 3, 3)[k % 5], limiter=k % 5 == 4,
                          solver=1 + 2 * (k % 3 == 0), cfl=0.3, bc=kinds(bc), **kw)


@pytest.mark.parametrize("n", [2, 3, 4, 5])
def test_alone(n, tslib):
    from turbostructred_gb300 import capi
    for k in range(30):
        out = []
        for tile in (None, (256, 1, 0)):
            with capi.Solver(case(n, k), precision=1) as s:
                if tile:
                    s.set_tile(*tile)
                s.set_state(wave(n, 1, 1))
                info, tm = s.step_timed(20)
                out.append((s.get_state(), info["time"]))
            assert list(tm["kernels"]) == ["k_mix_step" if tile else "k_tube32"]
        assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


def test_in_a_batch(tslib):
    """They do not take the set out of the tail mode: a few launches of many stages."""
    from turbostructred_gb300 import capi
    sizes, res = [2, 3, 500, 2, 64, 3, 4], []
    for tail in (True, False):
        with capi.Batch(16 << 20) as b:
            b.set_tail(tail)
            ids = [b.add(case(n, k, max_iter=60, max_time=1e30), wave(n, 1, 1)) for k, n in enumerate(sizes)]
            b.step(60)
            res.append(([b.get(i) for i in ids], b.stats()["launches"]))
    (a, few), (c, many) = res
    assert few <= len(sizes) and many >= 60
    for (u, i), (v, j) in zip(a, c):
        assert np.array_equal(u, v) and i["time"] == j["time"] and i["iteration"] == j["iteration"] == 60
