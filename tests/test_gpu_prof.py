"""Timing the launches (mhd_prof_enable) changes neither what is launched nor a
bit of the result; and the faces in one launch equal the faces in a launch per
direction, bit for bit, in every form: all nine variables, U and V, with every
limiter's end fills, both solvers and both schemes."""
import numpy as np
import pytest

from mhdcase import make_case

pytestmark = pytest.mark.gpu

FACES = ("flux_r", "flux_phi", "flux_z", "stage")


def steps(M, grid, p, U, V, n=2, **prof):
    d = M.Disc(grid, p)
    d.upload(U, V)
    if prof:
        d.prof(**prof)
    t, n0 = 0.0, d.launches()
    for _ in range(n):
        rc, t, *_ = d.step(t)
        assert rc == 0
    launches = d.launches() - n0
    kinds = {k: v[1] for k, v in d.prof_read().items()}
    out = d.download()
    d.close()
    return out, launches, kinds


def same(a, b):
    return all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b))


# one launch for the faces, and (superbee on a larger grid) one per direction
@pytest.mark.parametrize("case,dims,one", [("rk3_minmod_hlld", (14, 34, 130), True),
                                           ("rk2_superbee_hlld", (224, 224, 128), False)])
@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp32x2"])
def test_timed_steps_are_the_steps(M, case, dims, one, prec):
    if prec == "fp64":
        one = True
    grid, p, U, V = make_case(M, case, dims, precision=prec)
    plain, n0, _ = steps(M, grid, p, U, V, 1)
    timed, n1, kinds = steps(M, grid, p, U, V, 1, on=True)
    stages = 3 if case.startswith("rk3") else 2
    assert n0 == n1 and same(plain, timed)
    assert [kinds[k] for k in FACES] == ([0, 0, 0, stages] if one else [stages, stages, stages, 0])
    assert kinds["update"] == kinds["ghost"] == stages and kinds["setdt"] == 1


@pytest.mark.parametrize("dims", [(14, 6, 12), (17, 6, 97), (50, 82, 80)])
@pytest.mark.parametrize("case", ["rk3_minmod_hlld", "rk2_minmod_hlld", "rk3_minmod_hll", "rk3_mc_hlld_grav_cool",
                                  "rk2_vanleer_hlld_grav_cool", "rk3_superbee_hll_grav_cool", "rk2_superbee_hlld"])
@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp32x2"])
def test_one_launch_equals_a_launch_per_direction(M, dims, case, prec):
    grid, p, U, V = make_case(M, case, dims, precision=prec)
    one, n1, k1 = steps(M, grid, p, U, V)
    each, n3, k3 = steps(M, grid, p, U, V, on=True, by_direction=True)
    stages = 2 * (3 if case.startswith("rk3") else 2)
    assert n3 == n1 + 2 * stages and [k3[k] for k in FACES] == [stages, stages, stages, 0]
    assert same(one, each)
