"""Residual norms on the mixed 2D path: which kernel serves a domain with them, its bits and its norms."""
import numpy as np
import pytest

from test_flat2d import kinds, wave

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,norms,kernel", [(256, 256, 1, "k_flat2d"), (257, 256, 1, "k_mix_step"),
                                                (362, 362, 1, "k_mix_step"), (362, 362, 0, "k_flat2d"),
                                                (363, 362, 0, "k_mix_step")])
def test_kernel_and_norms(nx, ny, norms, kernel, tslib):
    """With norms the kernel that marches nothing gives way at half the cells (362^2: 38.2 us per stage against 25.4)."""
    from turbostructred_gb300 import capi
    case = capi.make_case(ndims=2, nx=nx, ny=ny, periodic=(1, 0, 1), recon=3, solver=3, cfl=0.4, bc=kinds("wall"),
                          residual_norms=bool(norms))
    ic, out = wave(nx, ny, 1), []
    for prec, tile in ((1, None), (1, (64, 1, 0)), (0, None)):
        with capi.Solver(case, precision=prec) as s:
            if tile:
                s.set_tile(*tile)
            s.set_state(ic)
            info, tm = s.step_timed(5)
            if prec == 1 and not tile:
                assert list(tm["kernels"]) == [kernel]
            out.append((s.get_state(), info))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1]["time"] == out[1][1]["time"]
    if norms:
        np.testing.assert_allclose(out[0][1]["residual"][:3], out[2][1]["residual"][:3], rtol=1e-4)
