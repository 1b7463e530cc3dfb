"""A NaN or an infinity outside the wet cells of a level that runs in the coarse tail:
the sweeps bring it to the wet cells, as they do on levels too large for the tail and
with the tail off (small_smooth = 0), and the solve says so."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")

CASES = {
    "2d5": dict(nx=16, ny=14, nz=1, case="twod"),
    "2d9-vertices": dict(nx=15, ny=16, nz=1, case="twod", location="vertices", operator="laplacian9"),
    "varcoef": dict(nx=16, ny=16, nz=1, case="twod", operator="varcoef"),
    "2d5-periodic": dict(nx=24, ny=18, nz=1, case="twod", topology="xperio"),
    "3d7": dict(nx=5, ny=5, nz=5, case="threed"),
    "3d19-vertices": dict(nx=5, ny=5, nz=5, case="threed", location="vertices", operator="laplacian9"),
}


def _solve(small, where, bad, fused=1, **p):
    rng = np.random.default_rng(1)
    mg = cfmg.get_gmg(cfmg.Param(verbose=False, cycle="v", npre=2, npost=2, omega=0.8, tol=1e-8, maxite=6, **p))
    mg.set_option("small_smooth", small)
    mg.set_option("fused_descent", fused)
    m = mg.download(1, "msk")
    land = (m.shape[0] // 2, m.shape[1] // 2, m.shape[2] // 2)
    m[land] = 0
    mg.oper[1].msk = m
    cfmg.setup_operators(mg)
    for lev in range(1, mg.nlevels + 1):
        for f in ("x", "y", "r", "b"):
            cfmg.set_to_zero(mg, lev, f)
    m = mg.download(1, "msk").astype(np.float64)
    b, x = rng.standard_normal(m.shape) * m, np.zeros(m.shape)
    if where == "b":
        b[land] = bad
    elif where == "x":
        x[land] = bad
    else:  # outside every sweep's range in 2D: read by the cells beside it
        x[m.shape[0] // 2, 0, 0] = bad
    mg.data[1].b, mg.data[1].x = b, x
    try:
        cfmg.solve(mg)
        return "finite"
    except cfmg.CfmgError as e:
        return "non-finite" if "non-finite" in str(e) else str(e)
    finally:
        mg.close()


@pytest.mark.parametrize("bad", [np.nan, -np.inf])
@pytest.mark.parametrize("where", ["b", "x", "edge"])
@pytest.mark.parametrize("name", list(CASES))
def test_nonfinite_on_land_ends_the_solve(name, where, bad):
    a, b = (_solve(small, where, bad, **CASES[name]) for small in (4, 0))
    assert a == b, (a, b)
    if where != "edge":
        assert a == "non-finite"


@pytest.mark.parametrize("where", ["b", "x", "edge"])
@pytest.mark.parametrize("op", [dict(), dict(location="vertices", operator="laplacian9"), dict(operator="varcoef")])
def test_nonfinite_on_land_ends_the_solve_in_steps(op, where):
    """Level 1 in one-launch steps (k_tbg.cu) and in the separate kernels (the 9-point operator reads no edge cell)."""
    a, b = (_solve(4, where, np.nan, fused, nx=72, ny=64, nz=1, case="twod", **op) for fused in (1, 0))
    assert a == b, (a, b)
    if where != "edge":
        assert a == "non-finite"
