"""How the fixed-point residual passes split their cells. The right-hand side
they make is exact and the 7-point wet mean a sum of integers, so the solution does not
depend on the split: tolerance zero between the 3D forms (even spans of wet
planes, a row a thread, strips of rows) and between skipping dry planes and
writing them; the residual norms differ by the order of FP64 additions of one
sign, bounded by 1e-12 for these sizes. In 2D the coded diagonal is read in
words: every remainder of a row's length by four, against the FP64 pass (whose
right-hand side differs by FP32 rounding: the same count of iterations, and
solutions as close as the residuals of 1e-10 allow)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")


def _mask(kind, sh, rng):
    i, j, k = (np.arange(n).reshape([-1 if a == b else 1 for b in range(3)]) for a, n in enumerate(sh))
    if kind == "basin":  # deep and shallow columns, tiles without a wet cell
        depth = sh[2] * (0.2 + 0.8 * np.cos(i / 9.0) ** 2 * np.cos(j / 7.0) ** 2)
        return (k < depth) & (i < 0.7 * sh[0]) & ~((i > 20) & (j > 16))
    if kind == "gaps":  # dry planes between wet ones, in some tiles
        return (k % 5 != 2) | (i < 33)
    if kind == "slab":  # one wet plane near the top of some tiles, the whole depth in one
        return ((k == sh[2] - 6) & (j < 20)) | ((i < 9) & (j > 40))
    return np.ones(sh, bool)


@pytest.mark.parametrize("location", ["centers", "vertices"])
@pytest.mark.parametrize("kind", ["basin", "gaps", "slab", "full"])
def test_planes(kind, location):
    out = []
    for rows, skip in ((2, 1), (2, 0), (1, 1), (0, 1)):
        mg = cfmg.get_gmg(cfmg.Param(nx=70, ny=52, nz=38, case="threed", location=location, npre=2, npost=2, omega=0.8,
                                     tol=0.0, maxite=4, residual_norm="l2", precision="mixed", verbose=False))
        sh = mg.shape(1)
        m = (mg.download(1, "msk") != 0) & _mask(kind, sh, None)
        mg.oper[1].msk = np.asfortranarray(m.astype(np.uint8))
        cfmg.setup_operators(mg)
        mg.set_option("staged_residual", rows)
        mg.set_option("skip_dry", skip)
        for lev in range(1, mg.nlevels + 1):
            for f in ("x", "y", "r", "b"):
                cfmg.set_to_zero(mg, lev, f)
        b = np.random.default_rng(4).standard_normal(sh) * m
        mg.data[1].b = b - m * (b.sum() / m.sum())
        _, _, hist = cfmg.solve(mg, history=True)
        out.append((hist, mg.data[1].x))
        mg.close()
    assert np.isfinite(out[0][0]).all()
    for h, x in out[1:]:
        assert np.array_equal(x, out[0][1])
        np.testing.assert_allclose(h, out[0][0], rtol=1e-12)


@pytest.mark.parametrize("operator", ["laplacian", "laplacian9"])
@pytest.mark.parametrize("nx,ny", [(91, 64), (92, 95), (93, 33), (94, 70)])
def test_rows(nx, ny, operator):
    out = []
    for on in (1, 0):
        mg = cfmg.get_gmg(cfmg.Param(nx=nx, ny=ny, nz=1, case="twod", operator=operator, npre=2, npost=2, omega=0.8,
                                     tol=1e-10, maxite=60, residual_norm="l2", precision="mixed", verbose=False))
        mg.set_option("int_residual", on)
        m = mg.download(1, "msk").astype(np.float64)
        b = np.random.default_rng(nx).standard_normal(mg.shape(1)) * m
        mg.data[1].b = b - m * (b.sum() / m.sum())
        res, n = cfmg.solve(mg)
        x = mg.data[1].x * m
        out.append((res, n, x - m * (x.sum() / m.sum())))
        mg.close()
    assert out[0][0] <= 1e-10 and out[0][1] == out[1][1]
    assert np.linalg.norm(out[0][2] - out[1][2]) <= 1e-8 * np.linalg.norm(out[1][2])
