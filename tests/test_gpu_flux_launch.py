"""The split stage's r, phi and z faces in one launch against the launch per
direction that timed runs use: the same operations per face, so the plain form
keeps its bits.  Runs of 1, 4 and 16 faces, rows, lines and runs that do not fill
their blocks."""
import numpy as np
import pytest

from mhdcase import make_case, rel_l1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(14, 6, 12), (14, 6, 31), (17, 6, 97), (14, 34, 130), (50, 82, 80), (129, 98, 95)])
@pytest.mark.parametrize("case,prec", [("rk3_minmod_hlld", "fp64"), ("rk3_minmod_hlld", "fp32"),
                                       ("rk3_minmod_hlld", "fp32x2"),
                                       ("rk3_superbee_hll_grav_cool", "fp64")])
def test_one_launch_against_three(M, dims, case, prec):
    grid, p, U, V = make_case(M, case, dims, precision=prec)
    out = []
    for timed in (False, True):
        d = M.Disc(grid, p)
        d.upload(U, V)
        if timed:
            d.prof(True)
        t = 0.0
        for _ in range(2):
            rc, t, *_ = d.step(t)
            assert rc == 0
        out.append(d.download()[0])
        d.close()
    if prec == "fp64":
        assert np.array_equal(out[0], out[1])
    else:   # order-one components; at most FP32 rounding of a few ulp per stage
        assert np.all(rel_l1(out[0], out[1])[[0, 2, 5, 7]] <= 2e-6)
