"""The resident kernel of 1D FP64 problems (csrc/ts_tube64.cu): bit for bit the oracle's steps at the sizes where
its split changes (one CTA, the last with a cell more or less, the largest that it takes and the first that it leaves
to the stage kernels)."""
import numpy as np
import pytest

NAT = (5, 0.0, (0.0, 0.0, 0.0), 0.0)
SYM = (1, 0.0, (0.0, 0.0, 0.0), 0.0)
MOVING = (2, 0.0, (0.3, 0.0, 0.0), 0.0)


def state(n, seed, transverse=False):
    r = np.random.default_rng(seed)
    x = (np.arange(n) + 0.5) / n
    rho = np.where(x < 0.4, 1.0, 0.125) * (1.0 + 0.02 * r.uniform(-1, 1, n) * (x > 0.6))
    p = np.where(x < 0.4, 1.0, 0.1)
    v = np.zeros((n, 3))
    v[:, 0] = np.where(x < 0.4, 0.2, 0.0)
    if transverse:
        v[:, 1] = 0.1 * (x > 0.5)
    return np.concatenate([rho[:, None], rho[:, None] * v, (p / 0.4 + 0.5 * rho * (v * v).sum(-1))[:, None]], -1).reshape(1, 1, n, 5)


def wave(n, transverse):
    x = (np.arange(n) + 0.5) / n
    rho, p = 1.0 + 0.1 * np.sin(6 * x), 1.0 + 0.05 * np.cos(9 * x)
    v = np.stack([0.2 * np.cos(5 * x), 0.1 * x * transverse, 0 * x], -1)
    return np.concatenate([rho[:, None], rho[:, None] * v, (p / 0.4 + 0.5 * rho * (v * v).sum(-1))[:, None]], -1).reshape(1, 1, n, 5)


def agree(case, ic, oracle_mod, steps):
    from turbostructred_gb300 import capi
    full = oracle_mod.embed(case, ic)
    ref, rinfo = oracle_mod.advance(case, full, steps)
    with capi.Solver(capi.make_case(**case)) as s:
        s.set_state(full, capi.LAYOUT_WITH_GHOSTS)
        s.step(steps // 2)
        info = s.step(steps - steps // 2)
        got = s.get_state(capi.LAYOUT_WITH_GHOSTS)
    assert np.array_equal(got, ref)
    assert info["time"] == rinfo["time"] and info["dt"] == rinfo["dt"] and info["iteration"] == steps
    np.testing.assert_allclose(info["residual"], rinfo["residual"], rtol=1e-12, atol=1e-300)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [4, 31, 59, 60, 61, 397, 1000, 4063, 4064, 4065])
@pytest.mark.parametrize("per", [0, 1])
def test_sizes(n, per, tslib, oracle_mod):
    from oracle import oracle as O
    agree(O.make_case(ndims=1, nx=n, periodic=(per, 1, 1), recon=3, solver=1, cfl=0.4, bc=[NAT] * 6), state(n, n), oracle_mod, 21)


@pytest.mark.gpu
@pytest.mark.parametrize("recon,lim", [(0, 0), (1, 0), (2, 0), (3, 0), (3, 1)])
@pytest.mark.parametrize("solver", [1, 3])
@pytest.mark.parametrize("bc", ["natural", "symmetry", "moving", "sources"])
def test_schemes(recon, lim, solver, bc, tslib, oracle_mod):
    from oracle import oracle as O
    kw = {"bc": [{"symmetry": SYM, "moving": MOVING}.get(bc, NAT)] * 6}
    if bc == "sources":
        kw.update(uniform_acceleration=(-0.3, 0.0, 0.0), eps=0.1 if solver == 1 else 0.0)
    # unlimited slopes turn a jump into negative densities (in the oracle too): a smooth wave for them
    ic = wave(131, bc != "natural") if recon == 1 or lim == 1 else state(131, 7, transverse=bc != "natural")
    agree(O.make_case(ndims=1, nx=131, periodic=(0, 1, 1), recon=recon, limiter=lim, solver=solver, cfl=0.4, **kw),
          ic, oracle_mod, 60)


@pytest.mark.gpu
def test_run_ends_where_the_oracle_does(tslib, oracle_mod):
    from oracle import oracle as O
    from turbostructred_gb300 import capi
    case = O.make_case(ndims=1, nx=200, periodic=(0, 1, 1), recon=0, solver=1, cfl=0.5, bc=[NAT] * 6)
    ic = state(200, 1)
    for kw in (dict(max_iter=17, max_time=1e30), dict(max_iter=10 ** 7, max_time=0.05)):
        with capi.Solver(capi.make_case(**dict(case, **kw))) as s:
            s.set_state(ic)
            info = s.run()
            again = s.run() if "max_iter" in kw and kw["max_iter"] == 10 ** 7 else None
            got = s.get_state(capi.LAYOUT_WITH_GHOSTS)
        k = info["iteration"] if again is None else again["iteration"]
        assert info["iteration"] == 17 or info["time"] >= 0.05
        ref, rinfo = oracle_mod.advance(case, oracle_mod.embed(case, ic), k)
        assert np.array_equal(got, ref)
        assert (info if again is None else again)["time"] == rinfo["time"]
