"""1D FP64 problems whose cells are physical while some face states are not: second-order slopes, formed variable by
variable, give a face a negative pressure, on its left or on its right only.  HLLC takes the other wave speed there
(fmin and fmax drop the NaN of the sound speed's root) and goes on.  Bit for bit the oracle's steps in the resident
kernel and, at 4065 cells, in the stage kernels."""
import numpy as np
import pytest

NAT = (5, 0.0, (0.0, 0.0, 0.0), 0.0)
# (density, velocity, pressure) on the left and on the right, reconstruction, limiter, sides of the faces in question
STREAMS = {
    "colliding": ((1.0, 20.0, 1.0), (1.0, -20.0, 1.0), 3, 0, "lr"),
    "colliding_vk": ((1.0, 20.0, 1.0), (1.0, -20.0, 1.0), 3, 1, "lr"),
    "colliding_cold": ((1.0, 3.0, 1e-3), (1.0, -3.0, 1e-3), 3, 0, "lr"),
    "colliding_cold_vk": ((1.0, 3.0, 1e-3), (1.0, -3.0, 1e-3), 3, 1, "lr"),
    "receding_eno2": ((1.0, -2.0, 0.4), (1.0, 2.0, 0.4), 2, 0, "lr"),
    "from_the_left": ((1.0, 2.0, 0.1), (1.0, 0.0, 0.1), 3, 0, "r"),
    "from_the_left_eno2": ((1.0, 2.0, 0.1), (1.0, 0.0, 0.1), 2, 0, "r"),
    "from_the_right": ((1.0, 0.0, 0.1), (1.0, -2.0, 0.1), 3, 0, "l"),
    "from_the_right_eno2": ((1.0, 0.0, 0.1), (1.0, -2.0, 0.1), 2, 0, "l"),
}
STEPS = 60


def problem(name, n):
    from oracle import oracle as O
    left, right, recon, lim, _ = STREAMS[name]
    x = (np.arange(n) + 0.5) / n
    rho, u, p = (np.where(x < 0.5, a, b) for a, b in zip(left, right))
    ic = np.stack([rho, rho * u, 0 * x, 0 * x, p / 0.4 + 0.5 * rho * u * u], -1).reshape(1, 1, n, 5)
    return O.make_case(ndims=1, nx=n, periodic=(0, 1, 1), recon=recon, limiter=lim, solver=3, cfl=0.4, bc=[NAT] * 6), ic


def pressure(w):
    return 0.4 * (w[..., 4] - 0.5 * (w[..., 1:4] ** 2).sum(-1) / w[..., 0])


def face_pressures(u, recon, lim):
    """Pressures left and right of the interior faces of the cells u (n, 5) of a uniform grid."""
    g = np.concatenate([u[:1], u, u[-1:]])
    lo, hi = u - g[:-2], g[2:] - u
    if recon == 2:
        d = 0.5 * np.where(np.abs(lo) < np.abs(hi), lo, hi)
    else:
        d = 0.25 * (lo + hi)
        top, low = np.maximum(np.maximum(g[:-2], g[2:]), u), np.minimum(np.minimum(g[:-2], g[2:]), u)
        un, eps2, lim_v = 0.5 * (top - low), (5.0 / len(u)) ** 3, np.ones_like(u)
        with np.errstate(all="ignore"):
            for s in (d, -d):
                a = np.where(s > 0, top, low) - u
                if lim == 0:
                    k = np.where(s != 0, np.minimum(1.0, a / s), 1.0)
                else:
                    a, q = a / un, s / un
                    k = np.where((s != 0) & (un > 0), (a * a + eps2 + 2 * q * a) / (a * a + 2 * q * q + a * q + eps2), 1.0)
                lim_v = np.minimum(lim_v, k)
        d = lim_v * d
    return pressure(u + d)[:-1], pressure(u - d)[1:]


@pytest.mark.parametrize("name", sorted(STREAMS))
def test_inputs_have_such_faces(name, oracle_mod):
    """The oracle stays physical, and faces with a negative pressure on one side occur."""
    case, ic = problem(name, 100)
    full, info, left, right = oracle_mod.embed(case, ic), None, 0, 0
    for _ in range(STEPS):
        u = full[0, 0, 1:-1]
        assert pressure(u).min() > 0 and u[:, 0].min() > 0
        pl, pr = face_pressures(u, case["recon"], case["limiter"])
        left += int(((pl < 0) & (pr > 0)).sum())
        right += int(((pr < 0) & (pl > 0)).sum())
        full, info = oracle_mod.advance(case, full, 1, info)
    assert (left > 0, right > 0) == ("l" in STREAMS[name][4], "r" in STREAMS[name][4])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [100, 397, 4064, 4065])
@pytest.mark.parametrize("name", sorted(STREAMS))
def test_hllc_takes_the_other_wave_speed(name, n, tslib, oracle_mod):
    from turbostructred_gb300 import capi
    case, ic = problem(name, n)
    ref, rinfo = oracle_mod.advance(case, oracle_mod.embed(case, ic), STEPS)
    assert np.isfinite(ref[0, 0, 1:-1]).all()
    with capi.Solver(capi.make_case(**case)) as s:
        s.set_state(ic)
        info = s.step(STEPS)
        got = s.get_state(capi.LAYOUT_WITH_GHOSTS)
    assert np.array_equal(got, ref)
    assert info["time"] == rinfo["time"] and info["dt"] == rinfo["dt"] and info["health"] == 0
