"""The passes of the mixed loop that make its FP32 right-hand side and add its
correction, four cells a thread and with integer conversions, on lengths of
every remainder of a block's 1024 cells and on right-hand sides whose values
span more than FP32's range (they round to subnormal values and to zero):
against the FP64 solve. Both end at a relative residual of 1e-11, which bounds
the relative difference by 1e-11 times the condition number, below 2e5 for the
five-point operators here (4 / (pi / 120)^2, times 10 for kappa's contrast)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")

OPS = {
    "varcoef": dict(operator="varcoef"),
    "xperio": dict(topology="xperio", location="vertices"),
    "unfused-residual": dict(location="vertices"),
    "unfused-residual-mean": dict(),
}


@pytest.mark.parametrize("name", list(OPS))
@pytest.mark.parametrize("nx,ny", [(120, 90), (118, 97), (98, 58)])
def test_mixed_passes(name, nx, ny):
    x = []
    for precision in ("mixed", "fp64"):
        mg = cfmg.get_gmg(cfmg.Param(nx=nx, ny=ny, nz=1, case="twod", verbose=False, npre=2, npost=2, omega=0.8,
                                     tol=1e-11, maxite=60, residual_norm="l2", precision=precision, **OPS[name]))
        mg.set_option("engine_cells", 600)
        if name.startswith("unfused"):
            mg.set_option("int_residual", 0)
        rng = np.random.default_rng(nx)
        sh = mg.shape(1)
        if name == "varcoef":
            mg.oper[1].kappa = np.exp(0.5 * rng.standard_normal(sh))
        cfmg.setup_operators(mg)
        for lev in range(1, mg.nlevels + 1):
            for f in ("x", "y", "r", "b"):
                cfmg.set_to_zero(mg, lev, f)
        m = mg.download(1, "msk").astype(np.float64)
        b = rng.standard_normal(sh) * 10.0 ** np.where(rng.random(sh) < 0.2, 0, -rng.integers(0, 60, sh)) * m
        mg.data[1].b = b if name in ("xperio", "unfused-residual") else b - m * (b.sum() / m.sum())
        res, n = cfmg.solve(mg)
        assert res <= 1e-11, (precision, res, n)
        v = mg.data[1].x * m
        x.append(v if name in ("xperio", "unfused-residual") else v - m * (v.sum() / m.sum()))
        mg.close()
    assert np.linalg.norm(x[0] - x[1]) <= 2e-6 * np.linalg.norm(x[1])
