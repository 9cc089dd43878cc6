"""The FP32 forms' device layout (rows of whole 32-slot groups, the nine
variables of a group together) at z extents on both sides of a group's edge:
what is uploaded comes back, the CFL cell is found where the plain form finds
it, and a step follows the plain form's."""
import numpy as np
import pytest

from mhdcase import make_case, rel_l1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [12, 29, 30, 31, 32, 33, 61, 62, 63, 64])
@pytest.mark.parametrize("prec", ["fp32", "fp32x2"])
def test_round_trip_cfl_cell_and_step(M, nz, prec):
    dims = (14, 6, nz)
    grid, p64, U, V = make_case(M, "rk3_minmod_hlld", dims)
    _, p32, _, _ = make_case(M, "rk3_minmod_hlld", dims, precision=prec)
    # one cell far above the rest, next to the row's end, decides dt
    V[3, 2, 4, nz] = 30.0
    U = M.vtou(grid, V)
    a, b = M.Disc(grid, p64), M.Disc(grid, p32)
    a.upload(U, V)
    b.upload(U, V)
    Ub, Vb = b.download()
    assert np.array_equal(Vb, V.astype(np.float32).astype(np.float64))
    if prec == "fp32":
        assert np.array_equal(Ub, U.astype(np.float32).astype(np.float64))
    else:
        assert np.all(np.abs(Ub - U) <= 2.0 ** -45 * np.abs(U))
    dt64, _, ijk64 = a.setdt()
    dt32, _, ijk32 = b.setdt()
    assert ijk32 == ijk64 == (2, 4, nz)
    assert abs(dt32 - dt64) <= 1e-6 * dt64
    a.step(0.0)
    b.step(0.0)
    # order-one components; FP32 rounding of a few ulp per stage
    err = rel_l1(b.download()[0], a.download()[0])[[0, 2, 5, 7]]
    assert np.all(err <= 2e-6), err
    a.close()
    b.close()
