"""ts_step_timed on 1D domains that are resident on chip: the kernel and the launches of ts_step, and its results."""
import numpy as np
import pytest

from test_flat2d import kinds, wave

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,kernel", [(0, "k_tube64"), (1, "k_tube32")])
@pytest.mark.parametrize("steps,launches", [(1, 1), (4096, 1), (4097, 2)])
def test_resident_launches(prec, kernel, steps, launches, tslib):
    from turbostructred_gb300 import capi
    case = capi.make_case(ndims=1, nx=100, periodic=(0, 1, 1), recon=3, solver=1, cfl=0.4, bc=kinds("symmetry"))
    out = []
    for timed in (True, False):
        with capi.Solver(case, precision=prec) as s:
            s.set_state(wave(100, 1, 1))
            info, tm = s.step_timed(steps) if timed else (s.step(steps), None)
            out.append((s.get_state(), info))
        if timed:
            assert list(tm["kernels"]) == [kernel] and tm["launches"] == launches
            assert 0 < tm["kernels"][kernel] <= tm["total_ms"] <= 1.0001 * launches * tm["kernels"][kernel]
    (a, ia), (b, ib) = out
    assert np.array_equal(a, b) and ia["iteration"] == ib["iteration"] == steps and ia["time"] == ib["time"]


def test_launched_stages_keep_theirs(tslib):
    """Larger 1D domains, and an explicit tile, are timed launch by launch."""
    from turbostructred_gb300 import capi
    kw = dict(ndims=1, periodic=(0, 1, 1), recon=3, solver=1, cfl=0.4, bc=kinds("symmetry"))
    for prec, n, tile, per in ((0, 4065, None, 5), (1, 8673, None, 1), (1, 100, (256, 1, 0), 1)):
        with capi.Solver(capi.make_case(nx=n, **kw), precision=prec) as s:
            if tile:
                s.set_tile(*tile)
            s.set_state(wave(n, 1, 1))
            info, tm = s.step_timed(3)
        assert info["iteration"] == 3 and tm["launches"] == 3 * per and len(tm["kernels"]) == per
        assert not any(k.startswith("k_tube") for k in tm["kernels"])
