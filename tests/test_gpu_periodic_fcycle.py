"""Mixed x-periodic cycles, whose blocked passes write the periodic images and leave out
the fills of fields that nothing reads, against one kernel per sweep with every fill
(temporal_blocking = 0, small_smooth = 0), bit for bit, V and F. Extents down to
levels narrower than the halo, through odd ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")


@pytest.mark.parametrize("pairs", [(2, 2), (1, 3), (0, 2), (2, 0)])
@pytest.mark.parametrize("cycle", ["v", "f"])
@pytest.mark.parametrize("size,nlevels", [((320, 192), 0), ((282, 150), 0), ((640, 64), 4), ((96, 500), 3)])
def test_periodic_cycles(size, nlevels, cycle, pairs):
    out = []
    for plain in (False, True):
        rng = np.random.default_rng(4)
        mg = cfmg.get_gmg(cfmg.Param(nx=size[0], ny=size[1], nz=1, case="twod", topology="xperio", operator="laplacian",
                                     cycle=cycle, npre=pairs[0], npost=pairs[1], omega=0.8, nlevels=nlevels,
                                     precision="mixed", residual_norm="l2", tol=0.0, maxite=5, verbose=False))
        if plain:
            mg.set_option("temporal_blocking", 0)
            mg.set_option("small_smooth", 0)
        m = mg.download(1, "msk")
        m[:, 3:-3] *= (rng.random(m[:, 3:-3].shape) > 0.02).astype(np.uint8)
        mg.oper[1].msk = m
        cfmg.fill(mg, 1, "msk")
        cfmg.setup_operators(mg)
        for lev in range(1, mg.nlevels + 1):
            for f in ("x", "y", "r", "b"):
                cfmg.set_to_zero(mg, lev, f)
        m = mg.download(1, "msk").astype(np.float64)
        b = rng.standard_normal(m.shape) * m
        mg.data[1].b = b - m * (b.sum() / m.sum())
        cfmg.fill(mg, 1, "b")
        _, _, hist = cfmg.solve(mg, history=True)
        out.append((hist, mg.data[1].x))
        mg.close()
    assert np.all(np.isfinite(out[0][0]))
    assert np.array_equal(out[0][0], out[1][0]), (out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
