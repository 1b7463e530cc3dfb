"""The FP64 operators on levels large enough for their test of all-zero warps
(half a million cells), against the oracle, sign bits of zeros included: land
covers most of the domain and holds zeros of either sign in x and b. The
operators are the same IEEE operations, so the tolerance is zero. NaN and Inf
on land reach the sweeps only (on a dry cell the masked residual is a select
here and a product in the oracle)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")

CASES = {
    "2d5": dict(nx=740, ny=716, nz=1, case="twod"),
    "2d9-vertices": dict(nx=728, ny=730, nz=1, case="twod", location="vertices", operator="laplacian9"),
    "varcoef": dict(nx=733, ny=725, nz=1, case="twod", operator="varcoef"),
    "3d7": dict(nx=86, ny=84, nz=70, case="threed"),
    "3d19-vertices": dict(nx=84, ny=86, nz=70, case="threed", location="vertices", operator="laplacian9"),
}


def _same_bits(a, b, what):
    ok = (a.view(np.int64) == b.view(np.int64)) | (np.isnan(a) & np.isnan(b))
    assert ok.all(), (what, int((~ok).sum()))


@pytest.mark.parametrize("omega", [0.8, 1.2])
@pytest.mark.parametrize("name", list(CASES))
def test_zero_operands(name, omega):
    p = dict(CASES[name], nlevels=2, omega=omega)
    og = O.OracleGmg(p)
    mg = cfmg.get_gmg(cfmg.Param(**p, verbose=False))
    rng = np.random.default_rng(2)
    shape = og.shape(1)
    i = np.arange(shape[0])[:, None, None]
    j = np.arange(shape[1])[None, :, None]
    wet = np.broadcast_to((i + j) % (shape[0] // 2) < shape[0] // 6, shape)  # diagonal bands, a third wet
    m = np.asfortranarray(wet.astype(np.uint8))
    if name == "varcoef":
        kap = np.asfortranarray(np.exp(0.5 * rng.standard_normal(shape)))
        og.field(1, "kappa")[...] = kap
        mg.oper[1].kappa = kap
    og.field(1, "msk")[...] = m
    og.setup_operators()
    mg.oper[1].msk = m
    cfmg.setup_operators(mg)

    def state(special):
        for lev in (1, 2):
            sh = og.shape(lev)
            mm = og.field(lev, "msk") != 0
            for f in ("x", "y", "b", "r"):
                a = np.asfortranarray(rng.standard_normal(sh))
                a[~mm] = np.where(rng.random(sh) < 0.5, -0.0, 0.0)[~mm]  # zeros of either sign, lane by lane
                if f != "b":
                    a[: sh[0] // 2][~mm[: sh[0] // 2]] = 0.0  # and long runs of +0
                if special and f in ("x", "b"):
                    land = np.flatnonzero(~mm.ravel(order="F"))
                    flat = a.ravel(order="F")
                    flat[rng.choice(land, 40, replace=False)] = rng.choice([np.nan, np.inf, -np.inf], 40)
                    a = np.asfortranarray(flat.reshape(sh, order="F"))
                og.field(lev, f)[...] = a
                mg.upload(lev, f, a)

    state(False)
    og.smooth(1, 1)
    mg.smoother[1](mg, 1, 1)
    _same_bits(og.field(1, "x"), mg.data[1].x, "smooth")
    _same_bits(og.field(1, "y"), mg.data[1].y, "smooth y")
    og.residual(1)
    mg.residual[1](mg, 1)
    _same_bits(og.field(1, "r"), mg.data[1].r, "residual")
    for f in ("r", "b"):
        og.restrict(1, f)
        mg.restriction[1](mg, 1, f)
        _same_bits(og.field(2, "b"), mg.data[2].b, "restrict")
    og.prolong(1)
    mg.prolongation[1](mg, 1)
    _same_bits(og.field(1, "x"), mg.data[1].x, "prolong")
    state(True)
    og.smooth(1, 1)
    mg.smoother[1](mg, 1, 1)
    _same_bits(og.field(1, "x"), mg.data[1].x, "smooth, non-finite land")
    _same_bits(og.field(1, "y"), mg.data[1].y, "smooth y, non-finite land")
    mg.close()
