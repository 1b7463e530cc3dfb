"""The coarse tail (one block in shared memory) against the same operators as
Ops of the cluster engine (option small_smooth = 0): every field of every
level, bit for bit. The two forms do the same additions in the same order, so
the tolerance is zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")


def _mask(shape, nh, rng):
    m = np.zeros(shape, dtype=np.uint8, order="F")
    sl = (slice(nh, -nh), slice(nh, -nh), slice(nh, -nh) if shape[2] > 2 * nh else slice(None))
    m[sl] = rng.random(m[sl].shape) > 0.025
    return m


def _state(mg):
    return {(lev, f): mg.download(lev, f) for lev in range(1, mg.nlevels + 1) for f in ("x", "y", "r", "b")}


def _setup(small, seed, **p):
    rng = np.random.default_rng(seed)
    mg = cfmg.get_gmg(cfmg.Param(verbose=False, **p))
    mg.set_option("small_smooth", small)
    mg.oper[1].msk = _mask(mg.shape(1), mg.param.nh, rng)
    cfmg.fill(mg, 1, "msk")
    if mg.param.operator == "varcoef":
        mg.oper[1].kappa = np.exp(0.5 * rng.standard_normal(mg.shape(1)))
    cfmg.setup_operators(mg)
    for lev in range(1, mg.nlevels + 1):
        for f in ("x", "y", "r", "b"):
            cfmg.set_to_zero(mg, lev, f)
    m = mg.download(1, "msk").astype(np.float64)
    b = rng.standard_normal(mg.shape(1)) * m
    b -= m * (b.sum() / m.sum())
    mg.data[1].b = b
    cfmg.fill(mg, 1, "b")
    return mg, rng


CASES = {
    "2d5": dict(nx=48, ny=36, nz=1, case="twod"),
    "2d5-odd": dict(nx=37, ny=29, nz=1, case="twod"),  # levels through odd extents, level 1 in the tail
    "2d5-layers": dict(nx=24, ny=20, nz=2, case="twod"),
    "2d9-vertices": dict(nx=40, ny=56, nz=1, case="twod", location="vertices", operator="laplacian9"),
    "2d5-periodic": dict(nx=48, ny=32, nz=1, case="twod", topology="xperio"),
    "2d5-periodic-narrow": dict(nx=28, ny=36, nz=1, case="twod", topology="xperio"),  # down to nx = 1 < nh
    "3d7-periodic": dict(nx=12, ny=16, nz=12, case="threed", topology="xperio"),
    "varcoef": dict(nx=44, ny=52, nz=1, case="twod", operator="varcoef"),
    "3d7": dict(nx=24, ny=20, nz=12, case="threed"),
    "3d19-vertices": dict(nx=20, ny=24, nz=16, case="threed", location="vertices", operator="laplacian9"),
}


@pytest.mark.parametrize("cycle", ["v", "f"])
@pytest.mark.parametrize("name", list(CASES))
def test_tail_cycle_is_bit_identical(name, cycle):
    out = []
    for small in (4, 0):
        mg, _ = _setup(small, 3, cycle=cycle, npre=2, npost=2, omega=0.8, **CASES[name])
        for _ in range(2):
            cfmg.normresidual(mg, 1.0)  # the F-cycle restricts level 1's r
            cfmg.cycle(mg)
        out.append(_state(mg))
        mg.close()
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k


@pytest.mark.parametrize("omega", [0.8, 1.2])
@pytest.mark.parametrize("name", list(CASES))
def test_tail_smoothing_of_any_x(name, omega):
    """x and y hold values in land and halo cells too, so a level sweeps its whole range; omega > 1 does anyway."""
    out = []
    for small in (4, 0):
        mg, rng = _setup(small, 4, npre=1, npost=1, omega=omega, **CASES[name])
        for lev in range(1, mg.nlevels + 1):
            for f in ("x", "y", "b"):
                mg.upload(lev, f, rng.standard_normal(mg.shape(lev)))
            mg.smoother[lev](mg, lev, 3)
        cfmg.vcycle(mg)
        out.append(_state(mg))
        mg.close()
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k


@pytest.mark.parametrize("name", ["2d5", "2d9-vertices", "2d5-periodic", "2d5-periodic-narrow", "varcoef", "3d7", "3d19-vertices"])
def test_tail_mixed_solve_is_bit_identical(name):
    out = []
    for small in (4, 0):
        mg, _ = _setup(small, 5, cycle="v", npre=2, npost=2, omega=0.8, precision="mixed", residual_norm="l2",
                       tol=1e-9, maxite=12, **CASES[name])
        res, nite, hist = cfmg.solve(mg, history=True)
        out.append((hist, mg.data[1].x))
        mg.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])


def test_tail_lists_follow_the_coefficients():
    """New masks on one handle: the lists are remade, also after a write through a coefficient's device address."""
    out = []
    for small in (4, 0):
        mg, rng = _setup(small, 6, cycle="v", npre=2, npost=2, omega=0.8, **CASES["2d5"])
        cfmg.cycle(mg)
        first = _state(mg)
        mg.oper[1].msk = _mask(mg.shape(1), 3, rng)
        cfmg.setup_operators(mg)
        for lev in range(1, mg.nlevels + 1):
            for f in ("x", "y", "r", "b"):
                cfmg.set_to_zero(mg, lev, f)
        mg.data[1].b = rng.standard_normal(mg.shape(1)) * mg.download(1, "msk")
        cfmg.cycle(mg)
        second = _state(mg)
        mg.field_ptr(3, "Pcoef")
        mg.oper[2].idiag = mg.oper[2].idiag * (rng.random(mg.shape(2)) > 0.3)
        cfmg.cycle(mg)
        out.append((first, second, _state(mg)))
        mg.close()
    for a, b in zip(*out):
        for k in a:
            assert np.array_equal(a[k], b[k]), k
