"""Runs that leave the physical states, on the FP64 path: what becomes infinite or NaN does so in the cells, variables
and steps in which it does in the oracle (transverse momenta of zero included), in the resident 1D kernel and in the
stage kernels."""
import numpy as np
import pytest

NAT = (5, 0.0, (0.0, 0.0, 0.0), 0.0)
# (density, velocity, pressure) on the left and on the right
STREAMS = {
    "colliding": ((1.0, 20.0, 1.0), (1.0, -20.0, 1.0)),
    "receding": ((1.0, -20.0, 0.4), (1.0, 20.0, 0.4)),
    "from_the_left": ((1.0, 20.0, 1.0), (1.0, 0.0, 1.0)),
    "at_rest_without_pressure": ((1.0, 0.0, 0.0), (1.0, 0.0, 0.0)),  # no wave speed anywhere: an infinite time step
}
GRIDS = {1: [(4, 1, 1), (100, 1, 1), (4065, 1, 1)], 2: [(100, 6, 1)], 3: [(60, 5, 4)]}


@pytest.mark.gpu
@pytest.mark.parametrize("size", [n for nd in GRIDS for n in GRIDS[nd]])
@pytest.mark.parametrize("solver", [1, 3])
@pytest.mark.parametrize("recon,lim", [(0, 0), (1, 0), (2, 0), (3, 0), (3, 1)])
@pytest.mark.parametrize("name", sorted(STREAMS))
def test_as_the_oracle(name, recon, lim, solver, size, tslib, oracle_mod):
    from oracle import oracle as O
    from turbostructred_gb300 import capi
    nx, ny, nz = size
    nd = 1 + (ny > 1) + (nz > 1)
    left, right = STREAMS[name]
    x = (np.arange(nx) + 0.5) / nx
    rho, u, p = (np.where(x < 0.5, a, b) for a, b in zip(left, right))
    row = np.stack([rho, rho * u, 0 * x, 0 * x, p / 0.4 + 0.5 * rho * u * u], -1)
    ic = np.ascontiguousarray(np.broadcast_to(row, (nz, ny, nx, 5)))
    case = O.make_case(ndims=nd, nx=nx, ny=ny, nz=nz, periodic=(0, 1, 1), recon=recon, limiter=lim, solver=solver, cfl=0.4,
                       bc=[NAT] * 6)
    inner = oracle_mod.interior_slices(case)
    for steps in (12, 120):
        ref, rinfo = oracle_mod.advance(case, oracle_mod.embed(case, ic), steps)
        with capi.Solver(capi.make_case(**case)) as s:
            s.set_state(ic)
            info = s.step(steps)
            got = s.get_state()
        for v in range(5):
            assert np.array_equal(got[..., v], ref[inner][..., v], equal_nan=True), (v, steps)
        assert np.array_equal(info["time"], rinfo["time"], equal_nan=True)
        assert np.array_equal(info["dt"], rinfo["dt"], equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(397, 1, 1), (60, 40, 1), (20, 18, 16)])
@pytest.mark.parametrize("recon,lim", [(1, 0), (2, 0), (3, 0), (3, 1)])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_oblique_streams(seed, recon, lim, size, tslib, oracle_mod):
    """Fields that vary along every axis: a slope that is not finite along one of them enters the samples of all."""
    from oracle import oracle as O
    from turbostructred_gb300 import capi
    nx, ny, nz = size
    nd = 1 + (ny > 1) + (nz > 1)
    r = np.random.default_rng(seed)
    z, y, x = np.meshgrid(*[(np.arange(n) + 0.5) / n - 0.5 for n in (nz, ny, nx)], indexing="ij")
    d = r.normal(size=3)
    side = d[0] * x + d[1] * y + d[2] * z > 0
    v = np.stack([np.where(side, a, b) * (k < nd) for k, (a, b) in enumerate(r.uniform(-15, 15, (3, 2)))], -1)
    rho, p = (np.where(side, *r.uniform(0.2, 3, 2)) for _ in range(2))
    ic = np.concatenate([rho[..., None], rho[..., None] * v, (p / 0.4 + 0.5 * rho * (v * v).sum(-1))[..., None]], -1)
    case = O.make_case(ndims=nd, nx=nx, ny=ny, nz=nz, periodic=(seed % 2, 1 if nd < 2 else seed % 2, 1), recon=recon,
                       limiter=lim, solver=1, cfl=0.4, bc=[NAT] * 6)
    for steps in (10, 40):
        ref, rinfo = oracle_mod.advance(case, oracle_mod.embed(case, ic), steps)
        with capi.Solver(capi.make_case(**case)) as s:
            s.set_state(ic)
            info = s.step(steps)
            got = s.get_state()
        assert np.array_equal(got, ref[oracle_mod.interior_slices(case)].reshape(got.shape), equal_nan=True)
        assert np.array_equal(info["time"], rinfo["time"], equal_nan=True)
