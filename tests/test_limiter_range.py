"""The FP32 Barth-Jespersen limiter at the end of FP32's range: a cell much wider than its neighbours (a joint of two
blocks) takes up to half of a jump as its slope, which can be above 2^126 where neighbouring values are below 2^128."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NAT = (5, 0.0, (0.0, 0.0, 0.0), 0.0)


def problem(nd, solver):
    from turbostructred_gb300 import capi
    shape = (4 if nd > 2 else 1, 5 if nd > 1 else 1, 81)
    u = np.zeros(shape + (5,))
    u[..., 0] = 8e37
    u[..., 4] = np.array([1.0] * 40 + [50.0] + [190.0] * 40) * 1e36
    case = capi.make_case(ndims=nd, nx=81, ny=shape[1], nz=shape[0], periodic=(0, 1, 1), recon=3, solver=solver, cfl=0.1,
                          blocks={0: [(0.0, 1.0, 40), (0.3, 1.0, 1), (0.7, 1.0, 40)]}, bc=[NAT] * 6, max_iter=4,
                          max_time=1e30)
    return case, u


def check(got, case, u):
    """FP32 fluxes of four steps: about 1e-8 of the fields from the FP64 path (the limiter at 0 instead: 1e-2)."""
    from turbostructred_gb300 import capi
    with capi.Solver(case) as s:
        s.set_state(u)
        info = s.step(4)
        ref = s.get_state()
    x, i = got
    assert i["health"] == info["health"] == 0 and i["iteration"] == 4
    assert abs(i["time"] - info["time"]) <= 1e-6 * info["time"]
    assert np.abs(x - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("nd,tile", [(1, None), (1, (256, 1, 0)), (2, None), (2, (64, 1, 0)), (3, None), (3, (32, 8, 0)),
                                     (3, (16, 16, 0))])
@pytest.mark.parametrize("solver", [1, 3])
def test_single_domains(nd, tile, solver, tslib):
    from turbostructred_gb300 import capi
    case, u = problem(nd, solver)
    with capi.Solver(case, precision=1) as s:
        if tile:
            s.set_tile(*tile)
        s.set_state(u)
        info = s.step(4)
        check((s.get_state(), info), case, u)


@pytest.mark.parametrize("nd", [1, 2])
@pytest.mark.parametrize("tail", [True, False])
@pytest.mark.parametrize("solver", [1, 3])
def test_batches(nd, tail, solver, tslib):
    from turbostructred_gb300 import capi
    case, u = problem(nd, solver)
    with capi.Batch(32 << 20) as b:
        b.set_tail(tail)
        i = b.add(case, u)
        b.run()
        check(b.get(i), case, u)
