"""The FP64 residual and its norm in one launch (levels of at most a cell a
thread of the norm) against the separate kernels, every operator, at sizes on
either side of a block and of the whole range: r (the cells out of the
residual's range keep theirs) and the norm are the same operations in the same
order, tolerance zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")

CASES = {
    "5": dict(operator="laplacian"),
    "9-vertices": dict(operator="laplacian9", location="vertices"),
    "varcoef": dict(operator="varcoef"),
    "7": dict(case="threed"),
    "19-vertices": dict(case="threed", operator="laplacian9", location="vertices"),
}


@pytest.mark.parametrize("name,size", [("5", (40, 37, 1)), ("5", (506, 506, 1)), ("9-vertices", (59, 43, 1)),
                                       ("9-vertices", (505, 505, 1)), ("varcoef", (301, 77, 1)), ("7", (58, 58, 58)),
                                       ("7", (21, 18, 12)), ("19-vertices", (33, 29, 21))])
def test_residual_and_norm(name, size):
    p = dict(dict(case="twod"), **CASES[name])
    mg = cfmg.get_gmg(cfmg.Param(nx=size[0], ny=size[1], nz=size[2], nlevels=2, verbose=False, **p))
    mg.set_option("engine_cells", 0)
    sh = mg.shape(1)
    assert np.prod(sh) <= 1 << 18
    rng = np.random.default_rng(size[0])
    m = (mg.download(1, "msk") != 0) & (rng.random(sh) < 0.8)
    mg.oper[1].msk = np.asfortranarray(m.astype(np.uint8))
    if name == "varcoef":
        mg.oper[1].kappa = np.exp(rng.standard_normal(sh))
    cfmg.setup_operators(mg)
    for f in ("x", "b"):
        mg.upload(1, f, np.asfortranarray(rng.standard_normal(sh)))
    r0 = np.asfortranarray(rng.standard_normal(sh))
    mg.upload(1, "r", r0)
    mg.residual[1](mg, 1)
    a = mg.data[1].r
    want = cfmg.norm(mg, 1, "r")
    mg.upload(1, "r", r0)
    got = cfmg.normresidual(mg, 3.0)
    b = mg.data[1].r
    assert np.array_equal(a.view(np.int64), b.view(np.int64))
    assert got == want / 3.0
    mg.close()
