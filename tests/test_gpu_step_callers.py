"""Calls whose levels do not take the one-launch steps (coefficients that the caller
bound, fields that were not zeroed after the setup, more pairs of sweeps than a
step has, single smoothing calls): their small levels run in the tail or the engine, so
they take no more launches than with the steps off (fused_descent = 0), and give
the same bits."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")


def _launches(mg):
    n = ctypes.c_longlong()
    mg._check(mg._L.cfmg_launch_count(mg.handle, ctypes.byref(n)))
    return n.value


def _make(route, fused, **p):
    rng = np.random.default_rng(3)
    p = dict(dict(nz=1, case="twod", cycle="v", npre=2, npost=2, omega=0.8, residual_norm="l2", verbose=False), **p)
    mg = cfmg.get_gmg(cfmg.Param(**p))
    mg.set_option("fused_descent", fused)
    if p.get("operator") == "varcoef":
        mg.oper[1].kappa = np.exp(0.3 * rng.standard_normal(mg.shape(1)))
    cfmg.setup_operators(mg)
    if route != "dirty":
        for lev in range(1, mg.nlevels + 1):
            for f in ("x", "y", "r", "b"):
                cfmg.set_to_zero(mg, lev, f)
    if route == "bound":
        for lev in range(1, mg.nlevels + 1):
            mg.bind_level(lev, **{f: mg.download(lev, f) for f in ("diag", "idiag", "Rcoef", "Pcoef")})
    m = mg.download(1, "msk").astype(np.float64)
    b = rng.standard_normal(m.shape) * m
    mg.data[1].b = b - m * (b.sum() / m.sum())
    cfmg.set_to_zero(mg, 1, "x")
    return mg


PROBLEMS = {
    "5": dict(nx=64, ny=64),
    "9-vertices": dict(nx=144, ny=112, location="vertices", operator="laplacian9"),
    "varcoef": dict(nx=72, ny=64, operator="varcoef"),
    "varcoef-mixed": dict(nx=288, ny=256, operator="varcoef", precision="mixed"),
}


@pytest.mark.parametrize("cycle", ["v", "f"])
@pytest.mark.parametrize("route", ["bound", "dirty", "pairs"])
@pytest.mark.parametrize("name", list(PROBLEMS))
def test_solve(name, route, cycle):
    p = dict(PROBLEMS[name], cycle=cycle)
    if route == "pairs":
        p.update(npre=4, npost=4)
    if route == "dirty" and name == "varcoef-mixed":
        pytest.skip("the FP32 steps need no zeroed FP64 fields")
    out = []
    for fused in (1, 0):
        mg = _make(route, fused, **p)
        n0 = _launches(mg)
        _, _, hist = cfmg.solve(mg, history=True, tol=0.0, maxite=4)
        out.append((_launches(mg) - n0, hist, mg.data[1].x))
        mg.close()
    assert out[0][0] <= out[1][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])


def test_single_smoothing_call():
    """38 x 38 cells of a handle whose cycles take steps there."""
    out = []
    for fused in (1, 0):
        mg = _make("zeroed", fused, nx=64, ny=64)
        mg.data[2].b = np.random.default_rng(5).standard_normal(mg.shape(2)) * mg.download(2, "msk")
        mg.smoother[2](mg, 2, 3)
        n0 = _launches(mg)
        mg.smoother[2](mg, 2, 3)
        out.append((_launches(mg) - n0, mg.download(2, "x")))
        mg.close()
    assert out[0][0] <= out[1][0]
    assert np.array_equal(out[0][1], out[1][1])
