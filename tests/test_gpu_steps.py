"""The one-launch descent and ascent steps of 2D levels (k_tbg.cu; FP64, and the
FP32 ones of the variable-coefficient operator) against
the separate kernels (option fused_descent = 0): every field of every level
after cycles, bit for bit: the same operations in the same order, tolerance
zero. Sizes put tile edges inside, at and beyond the array, on levels through
odd extents."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")


def _make(fused, nx, ny, seed, upload=None, **p):
    rng = np.random.default_rng(seed)
    mg = cfmg.get_gmg(cfmg.Param(nx=nx, ny=ny, nz=1, case="twod", verbose=False, **p))
    mg.set_option("fused_descent", fused)
    shape = mg.shape(1)
    i, j = np.arange(shape[0])[:, None, None] / shape[0], np.arange(shape[1])[None, :, None] / shape[1]
    wet = ((i - 0.5) ** 2 + (j - 0.45) ** 2 < 0.18) & (rng.random(shape) > 0.002)
    mg.oper[1].msk = np.asfortranarray(wet.astype(np.uint8))
    if p.get("operator") == "varcoef":
        mg.oper[1].kappa = np.exp(0.5 * rng.standard_normal(shape))
    cfmg.setup_operators(mg)
    for lev in range(1, mg.nlevels + 1):
        for f in ("x", "y", "r", "b"):
            cfmg.set_to_zero(mg, lev, f)
    m = mg.download(1, "msk").astype(np.float64)
    b = rng.standard_normal(shape) * m
    mg.data[1].b = b - m * (b.sum() / m.sum())
    if upload:
        mg.upload(2, upload, rng.standard_normal(mg.shape(2)))
    return mg


def _run(fused, *a, cycles=2, **p):
    mg = _make(fused, *a, **p)
    for _ in range(cycles):
        cfmg.normresidual(mg, 1.0)
        cfmg.cycle(mg)
    out = {(lev, f): mg.download(lev, f) for lev in range(1, mg.nlevels + 1) for f in ("x", "y", "r", "b")}
    res, nite, hist = cfmg.solve(mg, history=True, maxite=3, tol=0.0)
    out["hist"], out["x"] = hist, mg.data[1].x
    mg.close()
    return out


OPS = {
    "5": dict(operator="laplacian"),
    "5-vertices": dict(operator="laplacian", location="vertices"),
    "9-vertices": dict(operator="laplacian9", location="vertices"),
    "9": dict(operator="laplacian9"),
    "varcoef": dict(operator="varcoef"),
}


@pytest.mark.parametrize("cycle", ["v", "f"])
@pytest.mark.parametrize("name", list(OPS))
@pytest.mark.parametrize("size,pairs", [((224, 160), (2, 2)), ((333, 270), (1, 3)), ((514, 390), (3, 1))])
def test_steps_are_bit_identical(name, cycle, size, pairs):
    p = dict(cycle=cycle, npre=pairs[0], npost=pairs[1], omega=0.8, nlevels=6, **OPS[name])
    a, b = (_run(fused, *size, 7, **p) for fused in (1, 0))
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("cycle", ["v", "f"])
@pytest.mark.parametrize("name", list(OPS))
def test_first_level_step_of_any_x(name, cycle):
    """Level 1 in the steps: the caller's x holds values in land and halo cells."""
    p = dict(cycle=cycle, npre=2, npost=2, omega=0.8, nlevels=4, **OPS[name])
    out = []
    for fused in (1, 0):
        mg = _make(fused, 150, 118, 5, **p)
        mg.data[1].x = np.random.default_rng(2).standard_normal(mg.shape(1))
        cfmg.normresidual(mg, 1.0)
        cfmg.cycle(mg)
        out.append([mg.download(lev, f) for lev in range(1, mg.nlevels + 1) for f in ("x", "y", "r", "b")])
        mg.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("upload", ["x", "b"])
def test_values_outside_the_wet_interior_take_the_separate_kernels(upload):
    """A caller's values in a coarse field (halo and land included) are what the reference's cycle sees; a solve
    captured before them is captured again."""
    p = dict(cycle="v", npre=2, npost=2, omega=0.8, nlevels=6)
    out = []
    for fused in (1, 0):
        mg = _make(fused, 300, 220, 3, **p)
        cfmg.solve(mg, maxite=2, tol=0.0)
        mg.upload(2, upload, np.random.default_rng(1).standard_normal(mg.shape(2)))
        cfmg.solve(mg, maxite=2, tol=0.0)
        out.append([mg.download(lev, f) for lev in (1, 2, 3) for f in ("x", "y", "r", "b")])
        mg.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("cycle", ["v", "f"])
@pytest.mark.parametrize("size,pairs", [((470, 378), (2, 2)), ((661, 333), (3, 1)), ((392, 401), (1, 3)),
                                        ((222, 150), (2, 2))])
def test_mixed_varcoef_steps_are_bit_identical(cycle, size, pairs):
    """The first three sizes' level 1 takes the register form of the FP32 steps, the other levels the general one."""
    p = dict(operator="varcoef", cycle=cycle, npre=pairs[0], npost=pairs[1], omega=0.8, nlevels=6, precision="mixed",
             residual_norm="l2")
    out = []
    for fused in (1, 0):
        mg = _make(fused, *size, 9, **p)
        _, _, hist = cfmg.solve(mg, history=True, maxite=6, tol=0.0)
        out.append((hist, mg.data[1].x))
        mg.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("name,cycle,size,nlevels", [("5", "v", (300, 212), 2), ("5-vertices", "f", (520, 390), 3),
                                                     ("9-vertices", "f", (512, 512), 3), ("9", "v", (470, 330), 3),
                                                     ("varcoef", "v", (333, 270), 2)])
def test_long_smoothing_of_the_last_level(name, cycle, size, nlevels):
    """A hierarchy that ends above the tail's sizes smooths its last level in passes of several pairs."""
    p = dict(cycle=cycle, npre=2, npost=2, omega=0.8, nlevels=nlevels, **OPS[name])
    a, b = (_run(fused, *size, 3, **p) for fused in (1, 0))
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("size,pairs", [((1500, 1404), (2, 2)), ((1537, 1210), (3, 1))])
def test_fcycle_steps_of_several_waves_of_tiles(size, pairs):
    """The descent after an F-cycle's prolongation, on a level of some 1100 tiles and more where 304 are resident: every
    tile prolongs the coarse x as it was before the step, whichever tiles have finished, and a second run repeats."""
    p = dict(operator="varcoef", cycle="f", npre=pairs[0], npost=pairs[1], omega=0.8, nlevels=6, precision="mixed",
             residual_norm="l2")
    out = []
    for fused in (0, 1, 1):
        mg = _make(fused, *size, 13, **p)
        _, _, hist = cfmg.solve(mg, history=True, maxite=4, tol=0.0)
        out.append((hist, mg.data[1].x))
        mg.close()
    for hist, x in out[1:]:
        assert np.array_equal(out[0][0], hist)
        assert np.array_equal(out[0][1], x)
