"""The resident kernel of 1D mixed-precision problems (csrc/ts_tube32.cu) at the sizes where its split changes,
against the FP64 path and the stage kernels on the same problem, and in a batch with problems of very different
sizes in one launch."""
import numpy as np
import pytest

from test_flat2d import SIDES, kinds, wave

pytestmark = pytest.mark.gpu


def three(case, ic, steps):
    """(resident, stage kernels, FP64): states and infos."""
    from turbostructred_gb300 import capi
    out = []
    for prec, tile in ((1, None), (1, (256, 1, 0)), (0, None)):
        with capi.Solver(case, precision=prec) as s:
            if tile:
                s.set_tile(*tile)
            s.set_state(ic)
            s.step(steps // 2)
            info = s.step(steps - steps // 2)
            out.append((s.get_state(), info))
    (a, ia), (b, ib), (c, ic_) = out
    assert ia["health"] == 0 and ia["iteration"] == ib["iteration"] == ic_["iteration"] == steps
    # FP32 fluxes summed over a few steps: about 1e-6 of the fields from the FP64 path; the
    # same operations as the stage kernels
    for x, i in ((b, ib), (c, ic_)):
        assert abs(ia["time"] - i["time"]) <= 1e-6 * i["time"]
        assert np.abs(a - x).max() <= 1e-5 * np.abs(c).max()


@pytest.mark.parametrize("n", [4, 31, 59, 60, 61, 397, 1000, 4096, 8672, 8673])
@pytest.mark.parametrize("per", [0, 1])
def test_sizes(n, per, tslib):
    from turbostructred_gb300 import capi
    three(capi.make_case(ndims=1, nx=n, periodic=(per, 1, 1), recon=3, solver=1, cfl=0.4, bc=kinds("natural")),
          wave(n, 1, 1), 9)


@pytest.mark.parametrize("recon,lim", [(0, 0), (1, 0), (2, 0), (3, 0), (3, 1)])
@pytest.mark.parametrize("solver", [1, 3])
@pytest.mark.parametrize("bc", sorted(SIDES))
def test_schemes(recon, lim, solver, bc, tslib):
    from turbostructred_gb300 import capi
    kw = dict(uniform_acceleration=(0.1, 0.0, 0.0), external_force=(0.05, 0.02, 0.0)) if bc == "wall" else {}
    three(capi.make_case(ndims=1, nx=131, periodic=(0, 1, 1), recon=recon, limiter=lim, solver=solver,
                         eps=0.1 if solver == 1 else 0.0, cfl=0.3, bc=kinds(bc), **kw), wave(131, 1, 1), 12)


def test_run_and_snapshot_times(tslib):
    from turbostructred_gb300 import capi
    case = capi.make_case(ndims=1, nx=200, periodic=(0, 1, 1), recon=3, solver=1, cfl=0.5, max_iter=10 ** 7, max_time=0.1,
                          save_solution_time=0.03, bc=kinds("natural"))
    out = []
    for tile in (None, (256, 1, 0)):
        with capi.Solver(case, precision=1) as s:
            if tile:
                s.set_tile(*tile)
            s.set_state(wave(200, 1, 1))
            out.append((s.run(), s.get_state()))
    (a, ua), (b, ub) = out
    assert a["iteration"] == b["iteration"] and abs(a["time"] - b["time"]) < 1e-6
    assert abs(a["next_solution_time"] - b["next_solution_time"]) < 1e-12
    assert np.abs(ua - ub).max() <= 1e-5 * np.abs(ub).max()


def test_nonphysical_state_runs_on(tslib):
    """A single domain steps on through a non-physical state and reports it, as on the stage kernels."""
    from turbostructred_gb300 import capi
    case = capi.make_case(ndims=1, nx=100, periodic=(0, 1, 1), recon=0, solver=1, cfl=0.4, bc=kinds("natural"))
    ic = wave(100, 1, 1)
    ic[..., 50, 0] = -1.0
    with capi.Solver(case, precision=1) as s:
        s.set_state(ic)
        info = s.step(10)
    assert info["iteration"] == 10 and info["health"] != 0


@pytest.mark.parametrize("sizes", [(4, 5, 7, 4000), (8, 64, 129, 1000, 31), (8672,)])
def test_batch_of_mixed_sizes(sizes, tslib):
    from turbostructred_gb300 import capi
    res = []
    for tail in (True, False):
        with capi.Batch(64 << 20) as b:
            b.set_tail(tail)
            ids = [b.add(capi.make_case(ndims=1, nx=n, periodic=(k % 2, 1, 1), recon=3 * (k % 2), solver=1 + 2 * (k % 2),
                                        cfl=0.4, max_iter=15 + k, max_time=1e30, bc=kinds("symmetry")), wave(n, 1, 1))
                   for k, n in enumerate(sizes)]
            b.run()
            res.append([b.get(i) for i in ids])
    for (a, ia), (c, ic) in zip(*res):
        assert np.array_equal(a, c) and ia["time"] == ic["time"] and ia["iteration"] == ic["iteration"]


def test_unhealthy_tubes_among_many(tslib):
    """A tube that turns non-physical in a large set is stopped where the stage kernels' waits stop it: the same
    iteration, flags and state."""
    from turbostructred_gb300 import capi
    res = []
    for tail in (True, False):
        with capi.Batch(64 << 20) as b:
            b.set_tail(tail)
            ids = []
            for k in range(180):
                n = 64 + 5 * (k % 40)
                ic = wave(n, 1, 1)
                if k % 30 == 7:  # a strong rarefaction from the middle: no Roe solution
                    ic[0, 0, :n // 2, 1], ic[0, 0, n // 2:, 1] = -20.0, 20.0
                    ic[..., 4] = 0.02 + 0.5 * ic[..., 1] ** 2 / ic[..., 0]
                ids.append(b.add(capi.make_case(ndims=1, nx=n, periodic=(0, 1, 1), recon=3 * (k % 2), solver=1, cfl=0.5,
                                                max_iter=120, max_time=1e30, bc=kinds("natural")), ic))
            b.run()
            res.append([b.get(i) for i in ids])
    assert sum(i["health"] != 0 for _, i in res[1]) >= 3  # the inputs do what they are for
    for (a, ia), (c, ic) in zip(*res):
        assert (ia["iteration"], ia["health"]) == (ic["iteration"], ic["health"])
        assert np.array_equal(a, c, equal_nan=True)
        assert ia["time"] == ic["time"] or (np.isnan(ia["time"]) and np.isnan(ic["time"]))
