"""The 19-point level-1 residual in fixed point (k_resid_int19) against the
FP64-arithmetic form (int_residual = 0), at the edges of its 32 x 8 tiles and
of its plane runs.

First residual from a random x: both forms are within 21 roundings of 2^-53 of
terms below 6 |x| of the exact r at every cell, against r of the size of x, so
the norms agree to 1e-13; 1e-12 is asked. Solves to 1e-8: the same cycle
count, solutions within 1e-8 (the stopping residual) of each other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")


def _solve(int_res, nx, ny, nz, location, cycle, maxite, x0):
    rng = np.random.default_rng(11)
    mg = cfmg.get_gmg(cfmg.Param(nx=nx, ny=ny, nz=nz, case="threed", location=location, operator="laplacian9",
                                 cycle=cycle, omega=0.8, precision="mixed", residual_norm="l2", tol=1e-8,
                                 maxite=maxite, verbose=False))
    mg.set_option("int_residual", int_res)
    m = mg.download(1, "msk")
    m[3 + nx // 3, 3 + ny // 3, :] = 0  # a dry column
    mg.oper[1].msk = m
    cfmg.setup_operators(mg)
    for lev in range(1, mg.nlevels + 1):
        for f in ("x", "y", "r", "b"):
            cfmg.set_to_zero(mg, lev, f)
    m = mg.download(1, "msk").astype(np.float64)
    b = rng.standard_normal(m.shape) * m
    mg.data[1].b = b - m * (b.sum() / m.sum())
    if x0:
        mg.data[1].x = rng.standard_normal(m.shape) * m
    res, nite, hist = cfmg.solve(mg, history=True)
    x = mg.data[1].x * m
    if location == "centers":
        x -= m * (x.sum() / m.sum())
    mg.close()
    return hist, nite, x


@pytest.mark.parametrize("location", ["vertices", "centers"])
@pytest.mark.parametrize("shape", [(32, 8, 8), (33, 9, 12), (31, 23, 40), (64, 17, 26), (20, 34, 70), (96, 40, 12)])
def test_first_residual(shape, location):
    a = _solve(1, *shape, location, "v", 0, True)[0]
    b = _solve(0, *shape, location, "v", 0, True)[0]
    assert np.allclose(a, b, rtol=1e-12, atol=0), (a, b)


@pytest.mark.parametrize("cycle", ["v", "f"])
@pytest.mark.parametrize("shape", [(32, 32, 32), (48, 40, 24)])
def test_solve(shape, cycle):
    ha, na, xa = _solve(1, *shape, "vertices", cycle, 60, False)
    hb, nb, xb = _solve(0, *shape, "vertices", cycle, 60, False)
    assert na == nb and ha[-1] <= 1e-8
    assert np.linalg.norm(xa - xb) <= 1e-8 * np.linalg.norm(xb)
