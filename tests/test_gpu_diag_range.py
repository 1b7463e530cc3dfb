"""Mixed form on a diagonal that the caller chose: one too large for the 64-bit sums of
the fixed-point residual takes FP64 arithmetic (as int_residual = 0 does), one
that fits them stays. The first residual of a large x, whose terms add up: the
forms agree to the FP32 rounding of the right-hand side that the 2D ones sum, 2^-24."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")

CASES = {
    "5": (dict(nx=60, ny=44, nz=1, case="twod"), (4.0, 26.0, 27.0, 100.0)),
    "9": (dict(nx=60, ny=44, nz=1, case="twod", location="vertices", operator="laplacian9"), (3.0, 3.75, 4.0, 25.0)),
    "7": (dict(nx=24, ny=20, nz=16, case="threed"), (6.0, 24.0, 25.0, 100.0)),
    "19": (dict(nx=24, ny=20, nz=16, case="threed", location="vertices", operator="laplacian9"), (6.0, 8.75, 9.0, 25.0)),
}


@pytest.mark.parametrize("name,diag", [(n, d) for n, (_, ds) in CASES.items() for d in ds])
def test_first_residual(name, diag):
    out = []
    for int_res in (1, 0):
        mg = cfmg.get_gmg(cfmg.Param(precision="mixed", residual_norm="l2", tol=0.0, maxite=0, verbose=False,
                                     **CASES[name][0]))
        mg.set_option("int_residual", int_res)
        cfmg.setup_operators(mg)
        for lev in range(1, mg.nlevels + 1):
            for f in ("x", "y", "r", "b"):
                cfmg.set_to_zero(mg, lev, f)
        m = mg.download(1, "msk").astype(np.float64)
        i, j, k = np.indices(m.shape)
        mg.oper[1].diag = diag * m
        mg.data[1].b = 1.9 * (-1.0) ** (i + j + k) * m
        mg.data[1].x = 1.9 * (-1.0) ** (i + j + k) * m  # neighbours of the other sign
        _, _, hist = cfmg.solve(mg, history=True)
        out.append(hist[0])
        mg.close()
    assert abs(out[0] - out[1]) <= 1e-7 * out[1], out
