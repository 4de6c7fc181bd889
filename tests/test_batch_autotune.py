"""The autotuner on sets of 1D problems that the resident kernel serves: it times the stage kernels, whose tiles it
chooses."""
import numpy as np
import pytest

from test_flat2d import kinds, wave

pytestmark = pytest.mark.gpu


def test_tiles_of_a_set_in_tail_mode(tslib):
    """2400 tubes of 124 cells (one 128-thread tile each, 16 CTAs per SM): caps of two or one CTAs per SM, and 512
    threads for 124 cells, take one and a half to three times as long per stage, so none of them is ever chosen; the
    problems go on as without."""
    from turbostructred_gb300 import capi
    case = capi.make_case(ndims=1, nx=124, periodic=(0, 1, 1), recon=0, solver=1, cfl=0.4, max_iter=20, max_time=1e30,
                          bc=kinds("natural"))
    ic = wave(124, 1, 1)
    res = []
    for tune in (True, False):
        with capi.Batch(256 << 20) as b:
            ids = [b.add(case, ic) for _ in range(2400)]
            b.step(3)
            if tune:
                for _ in range(6):
                    tx, _, ctas = b.autotune(20)
                    assert tx in (0, 128, 256) and ctas == 0
            b.run()
            res.append([b.get(i) for i in ids[::600]])
    for (u, a), (v, c) in zip(*res):
        assert np.array_equal(u, v) and a["time"] == c["time"] and a["iteration"] == c["iteration"] == 20
