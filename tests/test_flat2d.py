"""Small 2D and 3D problems on the mixed path: the 2D kernel that marches nothing (csrc/ts_flat2d.cu) on both sides
of its tiles' edges and of the line where it gives way to the marching kernel, and short marches of the 3D one,
against the FP64 path on the same problem."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIDES = {"natural": 5, "symmetry": 1, "wall": 0, "moving": 2, "inlet": 3}


def wave(nx, ny, nz, w3=False):
    x, y, z = [(np.arange(n) + 0.5) / n for n in (nx, ny, nz)]
    Z, Y, X = np.meshgrid(z, y, x, indexing="ij")
    nd3 = nz > 1
    rho = 1.0 + 0.2 * np.sin(6 * X) * np.cos(5 * Y) + 0.1 * np.sin(4 * Z) * nd3
    p = 1.0 + 0.1 * np.cos(4 * X + 3 * Y) + 0.1 * np.cos(5 * Z) * nd3
    v = np.stack([0.3 * np.cos(5 * Y), 0.2 * np.sin(4 * X), 0.1 * np.cos(6 * X) * (1.0 if w3 else nd3)], -1)
    return np.concatenate([rho[..., None], rho[..., None] * v, (p / 0.4 + 0.5 * rho * (v * v).sum(-1))[..., None]], -1)


def both(case, ic, steps):
    """(mixed, FP64) states and infos; FP32 fluxes summed over a few steps agree to about 1e-6 of the fields."""
    from turbostructred_gb300 import capi
    out = []
    for prec in (capi.PRECISION_MIXED, capi.PRECISION_FP64):
        with capi.Solver(case, precision=prec) as s:
            s.set_state(ic)
            info = s.step(steps)
            out.append((s.get_state(), info))
    (a, ia), (b, ib) = out
    assert ia["health"] == 0 and ia["iteration"] == ib["iteration"] == steps
    assert abs(ia["time"] - ib["time"]) <= 1e-6 * ib["time"]
    assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max()
    return a


def kinds(bc):
    vel = (0.2, 0.1, 0.0) if bc in ("moving", "inlet") else (0.0, 0.0, 0.0)
    return [(SIDES[bc], 1.0, vel, 1.0)] * 6


@pytest.mark.parametrize("nx,ny", [(2, 2), (31, 3), (32, 4), (33, 5), (65, 9), (3, 130), (362, 362), (363, 362)])
@pytest.mark.parametrize("per", [(0, 0, 1), (1, 0, 1), (1, 1, 1)])
def test_2d_sizes(nx, ny, per, tslib):
    from turbostructred_gb300 import capi
    both(capi.make_case(ndims=2, nx=nx, ny=ny, periodic=per, recon=3, solver=1, cfl=0.4, bc=kinds("symmetry")),
         wave(nx, ny, 1), 5)


@pytest.mark.parametrize("recon,lim", [(0, 0), (1, 0), (2, 0), (3, 0), (3, 1)])
@pytest.mark.parametrize("solver", [1, 3])
@pytest.mark.parametrize("bc", sorted(SIDES))
def test_2d_schemes(recon, lim, solver, bc, tslib):
    from turbostructred_gb300 import capi
    kw = dict(uniform_acceleration=(0.1, -0.3, 0.0), external_force=(0.05, 0.0, 0.0)) if bc == "wall" else {}
    both(capi.make_case(ndims=2, nx=45, ny=14, periodic=(0, 0, 1), recon=recon, limiter=lim, solver=solver,
                        eps=0.1 if solver == 1 else 0.0, cfl=0.3, bc=kinds(bc), **kw), wave(45, 14, 1), 6)


def test_2d_residual_norms_and_marching_kernel(tslib):
    """The norms of both precisions, and the flat kernel against the marching one on the same problem."""
    from turbostructred_gb300 import capi
    case = capi.make_case(ndims=2, nx=75, ny=41, periodic=(1, 0, 1), recon=3, solver=3, cfl=0.4, bc=kinds("wall"),
                          residual_norms=True)
    ic, out = wave(75, 41, 1), []
    for prec, tile in ((1, None), (1, (132, 1, 0)), (0, None)):
        with capi.Solver(case, precision=prec) as s:
            if tile:
                s.set_tile(*tile)
            s.set_state(ic)
            info = s.step(7)
            out.append((s.get_state(), info))
    np.testing.assert_allclose(out[0][1]["residual"][:3], out[2][1]["residual"][:3], rtol=1e-4)
    assert np.abs(out[0][0] - out[1][0]).max() <= 1e-5 * np.abs(out[2][0]).max()
    assert abs(out[0][1]["time"] - out[1][1]["time"]) <= 1e-6 * out[1][1]["time"]


@pytest.mark.parametrize("n", [(2, 2, 2), (33, 9, 3), (17, 17, 5), (32, 32, 32), (97, 20, 13), (16, 70, 31)])
def test_3d_short_marches(n, tslib):
    from turbostructred_gb300 import capi
    for per in ((0, 0, 0), (1, 1, 1)):
        both(capi.make_case(ndims=3, nx=n[0], ny=n[1], nz=n[2], periodic=per, recon=3, solver=1, cfl=0.4,
                            bc=kinds("symmetry")), wave(*n), 5)


@pytest.mark.parametrize("sizes", [((40, 3),), ((64, 64), (130, 65), (33, 200)), ((300, 300),) * 40])
def test_batch_rows_per_item(sizes, tslib):
    """2D problems of a batch, whose items get shorter as the set gets smaller (problems that end one after the
    other), against each alone in a batch: the same bits whatever the split."""
    from turbostructred_gb300 import capi
    probs = [(capi.make_case(ndims=2, nx=n, ny=m, periodic=(k % 2, 0, 1), recon=3 * (k % 3 > 0), solver=1 + 2 * (k % 2),
                             cfl=0.4, max_iter=10 + 7 * k, max_time=1e30, bc=kinds("symmetry")), wave(n, m, 1))
             for k, (n, m) in enumerate(sizes[:8])] + \
            [(capi.make_case(ndims=2, nx=n, ny=m, periodic=(1, 1, 1), recon=0, solver=1, cfl=0.4, max_iter=9, max_time=1e30),
              wave(n, m, 1)) for n, m in sizes[8:]]
    with capi.Batch(512 << 20) as b:
        ids = [b.add(c, v) for c, v in probs]
        b.run()
        res = [b.get(i) for i in ids]
    for k in range(min(8, len(probs))):
        with capi.Batch(64 << 20) as b:
            i = b.add(*probs[k])
            b.run()
            got, info = b.get(i)
        assert info["iteration"] == 10 + 7 * k
        assert np.array_equal(got, res[k][0]) and info["time"] == res[k][1]["time"]


@pytest.mark.parametrize("tiny", [1e-300, 3e-39, 1.1e-38, -2e-320])
def test_tiny_momenta_are_zeros_in_fp32(tiny, tslib):
    """Momenta below FP32's normal range are zeros of the working copy, whatever their bits."""
    from turbostructred_gb300 import capi
    case = capi.make_case(ndims=2, nx=40, ny=9, periodic=(0, 0, 1), recon=3, solver=1, cfl=0.4, bc=kinds("wall"))
    out = []
    for m in (0.0, tiny):
        ic = wave(40, 9, 1)
        ic[..., 3] = m
        with capi.Solver(case, precision=1) as s:
            s.set_state(ic)
            s.step(5)
            out.append(s.get_state())
    assert np.array_equal(out[0][..., [0, 1, 2, 4]], out[1][..., [0, 1, 2, 4]])
    assert np.abs(out[1][..., 3]).max() <= 2 * abs(tiny)
