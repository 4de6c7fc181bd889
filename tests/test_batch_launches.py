"""Launches of a batch whose problems differ in size and solver, and the same bits however they are grouped."""
import numpy as np
import pytest

from test_flat2d import kinds, wave

pytestmark = pytest.mark.gpu
STAGES = 32


def case(nd, n, m, solver, recon):
    from turbostructred_gb300 import capi
    return capi.make_case(ndims=nd, nx=n, ny=m, periodic=(0, int(nd < 2), 1), recon=recon, solver=solver, cfl=0.4,
                          max_iter=10 ** 6, max_time=1e30, bc=kinds("symmetry"))


def run(probs, tile=None, tail=True):
    from turbostructred_gb300 import capi
    with capi.Batch(512 << 20) as b:
        b.set_tail(tail)
        if tile:
            b.set_tile(2, tile, 1, 0)
        ids = [b.add(c, u) for c, u in probs]
        b.step(STAGES)
        launches = b.stats()["launches"]
        return launches, [b.get(i) for i in ids]


def same(a, b):
    for (u, i), (v, k) in zip(a, b):
        assert np.array_equal(u, v) and i["time"] == k["time"] and i["iteration"] == k["iteration"] == STAGES


@pytest.mark.parametrize("sides", [(33, 60, 64, 92, 100, 128, 130, 200), (128,) * 8, (16, 500, 257)])
def test_2d_sets_take_one_tile(sides, tslib):
    """A stage is one launch per solver, and one that closes a long list."""
    probs = [(case(2, n, sides[-k], 1 + 2 * (k % 2), 3 * (k % 3 > 0)), wave(n, sides[-k], 1)) for k, n in enumerate(sides)]
    launches, got = run(probs)
    assert launches <= 3 * STAGES
    for tile in (64, 132):
        same(got, run(probs, tile)[1])


@pytest.mark.parametrize("sizes", [tuple(64 + 21 * k for k in range(22)), (30, 61, 125, 250, 600, 900, 1500, 2100, 3000, 4000),
                                   (4000,) * 9, (8600, 5)])
def test_1d_sets_in_few_launches(sizes, tslib):
    """Sets that run at once on the GPU: at most as many launches as there are streams for all stages."""
    probs = [(case(1, n, 1, 1 + 2 * (k % 2), 3 * (k % 3 > 0)), wave(n, 1, 1)) for k, n in enumerate(sizes)]
    launches, got = run(probs)
    assert launches <= 5
    same(got, run(probs, tail=False)[1])
