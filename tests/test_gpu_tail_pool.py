"""The device store of coarse-tail programs when it is full (2 MB: smoothing calls of 1050
different lengths on each of four levels pass it): later calls run in the cluster
engine and give the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")


def test_a_full_store_falls_back_to_the_engine():
    out = []
    for small in (4, 0):
        mg = cfmg.get_gmg(cfmg.Param(nx=32, ny=32, nz=1, case="twod", cycle="v", npre=1, npost=1, omega=0.8, nlevels=5,
                                     verbose=False))
        mg.set_option("small_smooth", small)
        cfmg.setup_operators(mg)
        fields = [(lev, f) for lev in range(1, mg.nlevels + 1) for f in ("x", "y", "r", "b")]
        for lev, f in fields:
            cfmg.set_to_zero(mg, lev, f)
        if small:
            for lev in range(2, mg.nlevels + 1):
                for nite in range(1, 1051):
                    mg.smoother[lev](mg, lev, nite)
        rng = np.random.default_rng(8)
        mg.data[1].b = rng.standard_normal(mg.shape(1)) * mg.download(1, "msk")
        cfmg.set_to_zero(mg, 1, "x")
        cfmg.cycle(mg)
        mg.smoother[2](mg, 2, 2000)
        res, nite, hist = cfmg.solve(mg, history=True, tol=0.0, maxite=3)
        out.append((hist, {k: mg.download(*k) for k in fields}))
        mg.close()
    assert np.array_equal(out[0][0], out[1][0])
    for k in fields:
        assert np.array_equal(out[0][1][k], out[1][1][k]), k
