"""A handle that is used again after a change of its mask: the solve gives what a new
handle gives, bit for bit, also where cells that were wet are dry now."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")

CASES = {
    "2d5": dict(nx=160, ny=128, nz=1, case="twod"),
    "2d9-vertices": dict(nx=144, ny=160, nz=1, case="twod", location="vertices", operator="laplacian9"),
    "2d5-periodic": dict(nx=160, ny=96, nz=1, case="twod", topology="xperio"),
    "varcoef": dict(nx=160, ny=144, nz=1, case="twod", operator="varcoef"),
    "3d7": dict(nx=64, ny=48, nz=40, case="threed"),
    "3d7-vertices": dict(nx=48, ny=64, nz=32, case="threed", location="vertices"),
    "3d19-vertices": dict(nx=48, ny=48, nz=32, case="threed", location="vertices", operator="laplacian9"),
}


def _mask(mg, radius):
    """The default mask, dry outside a column of this radius."""
    m = mg.download(1, "msk")
    i = (np.arange(m.shape[0]) - m.shape[0] / 2)[:, None, None] / m.shape[0]
    j = (np.arange(m.shape[1]) - m.shape[1] / 2)[None, :, None] / m.shape[1]
    return np.asfortranarray(m * (i * i + j * j < radius * radius)).astype(np.uint8)


def _prepare(mg, msk, seed):
    mg.oper[1].msk = msk
    cfmg.fill(mg, 1, "msk")
    cfmg.setup_operators(mg)
    _inputs(mg, seed)


def _inputs(mg, seed):
    rng = np.random.default_rng(seed)
    for lev in range(1, mg.nlevels + 1):
        for f in ("x", "y", "r", "b"):
            cfmg.set_to_zero(mg, lev, f)
    m = mg.download(1, "msk").astype(np.float64)
    b = rng.standard_normal(m.shape) * m
    b -= m * (b.sum() / m.sum())
    mg.data[1].b = b
    cfmg.fill(mg, 1, "b")


def _new(p, cycle, precision):
    mg = cfmg.get_gmg(cfmg.Param(verbose=False, cycle=cycle, npre=2, npost=2, omega=0.8, precision=precision,
                                 residual_norm="l2", tol=0.0, maxite=5, **p))
    if p.get("operator") == "varcoef":
        mg.oper[1].kappa = np.exp(0.3 * np.random.default_rng(0).standard_normal(mg.shape(1)))
    return mg


def _result(mg):
    res, nite, hist = cfmg.solve(mg, history=True)
    return hist, mg.data[1].x


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("cycle", ["v", "f"])
@pytest.mark.parametrize("name", list(CASES))
def test_solve_after_a_new_mask(name, cycle, precision):
    mg = _new(CASES[name], cycle, precision)
    wide, narrow = _mask(mg, 0.47), _mask(mg, 0.28)
    _prepare(mg, wide, 1)
    _result(mg)
    _prepare(mg, narrow, 2)
    a = _result(mg)
    mg.close()
    mg = _new(CASES[name], cycle, precision)
    _prepare(mg, narrow, 2)
    b = _result(mg)
    mg.close()
    assert np.array_equal(a[0], b[0]), (a[0], b[0])
    assert np.array_equal(a[1], b[1])


def test_batch_after_new_masks():
    p = cfmg.Param(nx=64, ny=64, nz=1, case="twod", location="centers", operator="laplacian", cycle="f", npre=2, npost=2,
                   omega=0.8, tol=0.0, maxite=5, residual_norm="l2", precision="mixed", verbose=False)
    sizes = [160, 96, 224]
    out = []
    for first in (0.47, None):
        batch = cfmg.Batch(p, sizes, sizes)
        for radius in (first, 0.28):
            if radius is None:
                continue
            for i in range(len(sizes)):
                mg = batch.instance(i)
                cfmg.set_default_msk(mg)
                _prepare(mg, _mask(mg, radius), i)
            batch.solve()
        out.append([batch.instance(i).data[1].x for i in range(len(sizes))])
        batch.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
