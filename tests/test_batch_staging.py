"""The page-locked staging buffer of a batch: what goes through it, and that a long problem does not make it grow."""
import numpy as np
import pytest

from test_flat2d import kinds, wave

pytestmark = pytest.mark.gpu


def page_locked():
    """Bytes of shared resident memory, which page-locked host memory is counted as."""
    with open("/proc/self/status") as f:
        for line in f:
            if line.startswith("RssShmem"):
                return 1024 * int(line.split()[1])
    pytest.skip("no RssShmem")


def test_a_long_problem_keeps_no_host_memory(tslib):
    """4 million cells have 96 MB of geometry; the batch keeps none of it on the host."""
    from turbostructred_gb300 import capi
    n = 4_000_000
    ic = np.zeros((1, 1, n, 5))
    ic[..., 0], ic[..., 4] = 1.0, 2.5
    kw = dict(ndims=1, periodic=(0, 1, 1), recon=0, solver=1, cfl=0.4, max_iter=2, max_time=1e30, bc=kinds("natural"))
    with capi.Batch(1 << 30) as b:
        i = b.add(capi.make_case(nx=100, **kw), wave(100, 1, 1))  # the buffers are made
        b.run()
        b.get(i)
        before = page_locked()
        i = b.add(capi.make_case(nx=n, **kw), ic)
        b.run()
        assert page_locked() - before < 16 << 20
        got, info = b.get(i)
    assert info["iteration"] == 2 and info["health"] == 0
    # a gas at rest, to FP32 rounding of its own fluxes
    assert np.abs(got - ic).max() <= 1e-6


@pytest.mark.parametrize("n", [10917, 10918, 10919, 60000])
def test_geometry_on_either_way(n, tslib):
    """Graded axes whose geometry goes through the buffer, and longer ones whose geometry is copied by itself, against
    the same problem as a single domain (FP32 fluxes of a few steps)."""
    from turbostructred_gb300 import capi
    case = capi.make_case(ndims=1, nx=n, periodic=(0, 1, 1), recon=3, solver=3, cfl=0.4, max_iter=4, max_time=1e30,
                          blocks={0: [(0.0, 1.0 + 2.0 / n, n)]}, bc=kinds("symmetry"))
    ic = wave(n, 1, 1)
    with capi.Batch(64 << 20) as b:
        ids = [b.add(case, ic) for _ in range(2)]
        b.run()
        (u, a), (v, c) = [b.get(i) for i in ids]
    with capi.Solver(case, precision=1) as s:
        s.set_state(ic)
        info = s.step(4)
        w = s.get_state()
    assert np.array_equal(u, v) and a["iteration"] == c["iteration"] == 4
    assert abs(a["time"] - info["time"]) <= 1e-6 * info["time"]
    assert np.abs(u - w).max() <= 1e-5 * np.abs(w).max()
