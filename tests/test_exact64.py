"""The FP64 path's integer division and square root (csrc/ts_exact64.cuh):
bit for bit those of the hardware for every operand they accept, and the
kernels take the hardware operation for those they refuse."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "turbostructred_gb300", "csrc")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("x64") / "exact64_check")
    subprocess.run(["g++", "-O2", "-std=c++20", "-ffp-contract=off", "-I" + CSRC,
                    os.path.join(ROOT, "tests", "exact64_check.cpp"), "-o", exe], check=True)
    return exe


def _doubles(sign, exp, mant):
    return (sign.astype(np.uint64) << np.uint64(63) | exp.astype(np.uint64) << np.uint64(52) |
            mant.astype(np.uint64)).view(np.float64)


def operands(kind, n=400_000):
    r = np.random.default_rng(7)
    one = 1 << 52
    sgn = lambda: r.integers(0, 2, n)  # noqa: E731
    rnd = lambda: r.integers(0, one, n)  # noqa: E731
    near = lambda: np.where(r.integers(0, 2, n) == 0, r.integers(0, 9, n), one - 1 - r.integers(0, 9, n))  # noqa: E731
    e = lambda lo=513, hi=1534: r.integers(lo, hi, n)  # noqa: E731
    if kind == "random":
        return _doubles(sgn(), e(), rnd()), _doubles(sgn(), e(), rnd())
    if kind == "near_powers":
        return _doubles(sgn(), e(), near()), _doubles(sgn(), e(), near())
    if kind == "near_midpoints":
        # a within an ulp of (m + 1/2) b for a random 53-bit m; b also next to (m + 1/2)^2
        m, B = rnd() + one, rnd() + one
        a = (((2 * m + 1).astype(object) * B.astype(object)) >> 54).astype(np.float64)
        a = (a.view(np.int64) + r.integers(-1, 2, n)).view(np.float64)
        half = n // 2
        sq = ((m.astype(object) * m.astype(object) + m.astype(object)) >> 53).astype(np.float64) * 2.0
        b = B.astype(np.float64)
        b[half:] = (sq.view(np.int64) + r.integers(-1, 2, n)).view(np.float64)[half:]
        return a, b
    if kind == "zero_dividends":
        return np.where(sgn() == 0, 0.0, -0.0), _doubles(sgn(), e(), rnd())
    assert kind == "all_patterns"  # any bit pattern: subnormals, infinities, NaN, extreme exponents
    return _doubles(sgn(), r.integers(0, 2048, n), rnd()), _doubles(sgn(), r.integers(0, 2048, n), rnd())


@pytest.mark.parametrize("kind", ["random", "near_powers", "near_midpoints", "zero_dividends", "all_patterns"])
def test_quotients_and_roots_are_correctly_rounded(kind, checker):
    a, b = operands(kind)
    out = subprocess.run([checker], input=np.stack([a, b], 1).tobytes(), capture_output=True, check=True).stdout
    quo, rt, hf, refused = (int(x) for x in out.split())
    assert (quo, rt, hf) == (0, 0, 0)
    # finite operands in the stated ranges are never refused
    assert (refused == 0) == (kind != "all_patterns")


SYM = (1, 0.0, (0.0, 0.0, 0.0), 0.0)
NAT = (5, 0.0, (0.0, 0.0, 0.0), 0.0)


def kernel_cases():
    from oracle import oracle as O
    out = []
    for recon, lim in ((3, 0), (3, 1), (2, 0), (1, 0)):
        # a stretched periodic axis: ghost cells differ in size from the cells
        # they repeat, so slopes and limiters are kept apart (fold = 0)
        out.append((f"stretched_periodic_r{recon}l{lim}", 1.0, None,
                    O.make_case(ndims=2, nx=37, ny=29, periodic=(1, 0, 1), recon=recon, limiter=lim, cfl=0.3,
                                blocks={0: [(0.0, 1.04, 37)]}, bc=[NAT] * 6)))
    for solver in (1, 3):
        # operands outside the integer routines' ranges: the hardware's division everywhere, or at some faces
        out.append((f"tiny_state_s{solver}", 2.0 ** -520, None,
                    O.make_case(ndims=2, nx=33, ny=17, periodic=(1, 1, 1), recon=3, solver=solver, cfl=0.4)))
        out.append((f"tiny_transverse_s{solver}", 1.0, 1e-190,
                    O.make_case(ndims=2, nx=70, ny=19, periodic=(0, 1, 1), recon=3, solver=solver, cfl=0.4, bc=[SYM] * 6)))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("spec", kernel_cases(), ids=lambda s: s[0])
def test_kernels_outside_the_fast_ranges(spec, tslib, oracle_mod):
    name, scale, w, case = spec
    from turbostructred_gb300 import capi
    ic = capi.fill_scenario(capi.make_case(**case), 1, 11, [2.0, 1.0, 0.5, 2.5, 0.01]) * scale
    if w is not None:
        ic[..., ::3, 3] = w * ic[..., ::3, 0]
    full = oracle_mod.embed(case, ic)
    ref, rinfo = oracle_mod.advance(case, full, 9)
    with capi.Solver(capi.make_case(**case)) as s:
        s.set_state(full, capi.LAYOUT_WITH_GHOSTS)
        info = s.step(9)
        got = s.get_state(capi.LAYOUT_WITH_GHOSTS)
    assert np.array_equal(got, ref)
    assert info["time"] == rinfo["time"] and info["dt"] == rinfo["dt"]


@pytest.mark.parametrize("kind", ["random", "near_powers", "ties", "zero_dividends", "all_patterns"])
def test_products_are_correctly_rounded(kind, tmp_path):
    exe = str(tmp_path / "mul_check")
    subprocess.run(["g++", "-O2", "-std=c++20", "-ffp-contract=off", "-I" + CSRC,
                    os.path.join(ROOT, "tests", "exact64_mul_check.cpp"), "-o", exe], check=True)
    if kind == "ties":  # short significands: products of exactly 54 bits, and exact ones
        r = np.random.default_rng(3)
        a, b = (r.integers(1 << 26, 1 << 27, 400_000).astype(np.float64) for _ in range(2))
    else:
        a, b = operands(kind)
    out = subprocess.run([exe], input=np.stack([a, b], 1).tobytes(), capture_output=True, check=True).stdout
    wrong, refused = (int(x) for x in out.split())
    assert wrong == 0
    assert (refused == 0) == (kind != "all_patterns")


@pytest.mark.gpu
@pytest.mark.parametrize("scale,w", [(1.0, None), (2.0 ** -520, None), (1.0, 1e-190)], ids=["usual", "tiny_state", "tiny_w"])
@pytest.mark.parametrize("eps", [0.0, 0.1])
def test_3d_roe_faces(scale, w, eps, tslib, oracle_mod):
    """The 3D Roe faces, whose products run on the integer pipe, on sizes that leave partial warps and blocks."""
    from oracle import oracle as O
    from turbostructred_gb300 import capi
    case = O.make_case(ndims=3, nx=13, ny=7, nz=5, periodic=(1, 0, 0), recon=3, solver=1, eps=eps, cfl=0.4, bc=[SYM] * 6)
    r = np.random.default_rng(5)
    rho, p = r.uniform(0.5, 2.0, (5, 7, 13)), r.uniform(0.5, 2.0, (5, 7, 13))
    v = r.uniform(-0.5, 0.5, (5, 7, 13, 3)) * (r.uniform(size=(5, 7, 13, 1)) < 0.7)
    if w is not None:
        v[..., 2] = w
    ic = np.concatenate([rho[..., None], rho[..., None] * v, (p / 0.4 + 0.5 * rho * (v * v).sum(-1))[..., None]], -1) * scale
    full = oracle_mod.embed(case, ic)
    ref, rinfo = oracle_mod.advance(case, full, 6)
    with capi.Solver(capi.make_case(**case)) as s:
        s.set_state(full, capi.LAYOUT_WITH_GHOSTS)
        info = s.step(6)
        got = s.get_state(capi.LAYOUT_WITH_GHOSTS)
    assert np.array_equal(got, ref)
    assert info["time"] == rinfo["time"] and info["dt"] == rinfo["dt"]


@pytest.mark.gpu
@pytest.mark.parametrize("ndims", [2, 3])
@pytest.mark.parametrize("solver", [1, 3])
@pytest.mark.parametrize("recon", [0, 2, 3])
def test_waves_that_reach_far_into_still_gas(ndims, solver, recon, tslib, oracle_mod):
    """The transverse momentum ahead of a wave falls through all exponents down to zero: operands, products and quotients that are
    tiny, subnormal or vanish, in every kernel of the path."""
    from oracle import oracle as O
    from turbostructred_gb300 import capi
    n = {2: (150, 61, 1), 3: (60, 9, 11)}[ndims]
    case = O.make_case(ndims=ndims, nx=n[0], ny=n[1], nz=n[2], periodic=tuple(int(a >= ndims) for a in range(3)), recon=recon,
                       solver=solver, cfl=0.4, bc=[SYM] * 6)
    rho, p = np.ones(n[::-1]), np.full(n[::-1], 0.1)
    p[:n[2] // 2 + 1, :n[1] // 2 + 1, :9] = 10.0
    ic = np.zeros(n[::-1] + (5,))
    ic[..., 0], ic[..., 4] = rho, p / 0.4
    full = oracle_mod.embed(case, ic)
    ref, rinfo = oracle_mod.advance(case, full, 40)
    with capi.Solver(capi.make_case(**case)) as s:
        s.set_state(full, capi.LAYOUT_WITH_GHOSTS)
        info = s.step(40)
        got = s.get_state(capi.LAYOUT_WITH_GHOSTS)
    mom = np.abs(ref[..., 1:4])
    assert mom[mom > 0].min() < 1e-100  # the inputs do what they are for
    assert np.array_equal(got, ref) and info["time"] == rinfo["time"]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["diagonal", "linear", "ulps", "offset", "random", "almost_diagonal"])
@pytest.mark.parametrize("ndims", [2, 3])
def test_limiter_ties(kind, ndims, tslib, oracle_mod):
    """Slopes and limits that are equal, a few ulps apart or lost in the value's rounding: the limiter's smallest ratio is
    the reference's whichever way it is found."""
    from oracle import oracle as O
    from turbostructred_gb300 import capi
    n = (37, 37, 1) if ndims == 2 else (13, 13, 13)
    r = np.random.default_rng(11)
    x, y, z = [(np.arange(k) + 0.5) / k for k in n]
    Z, Y, X = np.meshgrid(z, y, x, indexing="ij")
    d = X + Y + (Z if ndims == 3 else 0.0)
    f = {"diagonal": 0.3 * np.sin(7 * d), "linear": 0.25 * d, "ulps": r.integers(-2, 3, X.shape) * 2.0 ** -52,
         "offset": 1e-9 * np.sin(9 * X) * np.cos(5 * Y), "random": 0.2 * r.uniform(-1, 1, X.shape),
         "almost_diagonal": 0.3 * np.sin(7 * d) * (1 + 1e-6 * r.uniform(-1, 1, X.shape))}[kind]
    rho, p = 1.0 + f, 1.0 + 0.5 * f
    v = np.stack([0.1 + f, 0.1 + f, (0.1 + f) * (ndims == 3)], -1)
    ic = np.concatenate([rho[..., None], rho[..., None] * v, (p / 0.4 + 0.5 * rho * (v * v).sum(-1))[..., None]], -1)
    case = O.make_case(ndims=ndims, nx=n[0], ny=n[1], nz=n[2], periodic=(1, 1, 1), recon=3, solver=3, cfl=0.3)
    full = oracle_mod.embed(case, ic)
    ref, rinfo = oracle_mod.advance(case, full, 7)
    with capi.Solver(capi.make_case(**case)) as s:
        s.set_state(full, capi.LAYOUT_WITH_GHOSTS)
        info = s.step(7)
        got = s.get_state(capi.LAYOUT_WITH_GHOSTS)
    assert np.isfinite(ref).all()
    assert np.array_equal(got, ref) and info["time"] == rinfo["time"]
