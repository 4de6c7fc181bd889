"""Grids graded so strongly that cells are narrower than the last bit of their coordinates: the distance of two
centres is zero there, and the slope of a constant state 0 / 0, in the FP64 kernels as in the oracle."""
import numpy as np
import pytest

NAT = (5, 0.0, (0.0, 0.0, 0.0), 0.0)


@pytest.mark.gpu
@pytest.mark.parametrize("n,q", [(600, 0.9), (4064, 0.985), (4065, 0.985)])
@pytest.mark.parametrize("recon,lim", [(1, 0), (2, 0), (3, 0), (3, 1)])
@pytest.mark.parametrize("per", [0, 1])
def test_distances_of_zero(n, q, recon, lim, per, tslib, oracle_mod):
    from oracle import oracle as O
    from turbostructred_gb300 import capi
    case = O.make_case(ndims=1, nx=n, periodic=(per, 1, 1), recon=recon, limiter=lim, solver=1, cfl=0.4,
                       blocks={0: [(0.0, q, n)]}, bc=[NAT] * 6)
    x = oracle_mod.grid(case)[0]
    assert (np.diff(x) == 0).any()
    ic = np.zeros((1, 1, n, 5))
    ic[..., 0], ic[..., 4] = np.where(x[1:-1] < 0.5, 1.0, 0.5), np.where(x[1:-1] < 0.5, 2.5, 1.0)
    for steps in (1, 4):
        ref, rinfo = oracle_mod.advance(case, oracle_mod.embed(case, ic), steps)
        with capi.Solver(capi.make_case(**case)) as s:
            s.set_state(ic)
            info = s.step(steps)
            got = s.get_state()
        assert np.array_equal(got[0, 0], ref[0, 0, 1:-1], equal_nan=True)
        assert np.array_equal(info["time"], rinfo["time"], equal_nan=True)
