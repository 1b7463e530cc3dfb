"""The start of a batched solve (k_binit): a cluster of blocks per instance, of which
all but the first hold almost no cells on instances as small as these. Copies of
one problem, wherever they stand in the batch, start from the same |b| and range,
so they return the same bits, solve after solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")


def _setup(g, seed):
    rng = np.random.default_rng(seed)
    cfmg.set_default_msk(g)
    cfmg.setup_operators(g)
    for lev in range(1, g.nlevels + 1):
        for f in ("x", "y", "r", "b"):
            cfmg.set_to_zero(g, lev, f)
    m = g.download(1, "msk").astype(np.float64)
    b = rng.standard_normal(m.shape) * m
    g.data[1].b = b - m * (b.sum() / m.sum())


def test_copies_of_tiny_instances_return_the_same_bits():
    sizes = [8, 16, 12] * 100
    p = cfmg.Param(nx=8, ny=8, nz=1, case="twod", location="centers", operator="laplacian", cycle="v", npre=2, npost=2,
                   omega=0.8, tol=1e-10, maxite=30, residual_norm="l2", precision="mixed", verbose=False)
    batch = cfmg.Batch(p, sizes, sizes)
    for i, n in enumerate(sizes):
        _setup(batch.instance(i), n)
    first = None
    for _ in range(4):
        res, nite, _ = batch.solve()
        assert np.all(res <= 1e-10) and np.all(nite > 0)
        x = [batch.instance(i).data[1].x for i in range(len(sizes))]
        for i in range(len(sizes)):
            assert res[i] == res[i % 3] and nite[i] == nite[i % 3] and np.array_equal(x[i], x[i % 3]), i
        first = first or (list(res[:3]), x[:3])
        assert first[0] == list(res[:3]) and all(np.array_equal(a, c) for a, c in zip(first[1], x))
    batch.close()
