"""The FP64 9-point sweep and residual of large levels, whose sums of
neighbours are integer ones, against the oracle: extents at the edges of the
30 x 16 cells that a block takes, and fields that reach each branch (sums that
round, that tie, that cancel, values too far apart for the integers, zeros of
either sign, subnormal and non-finite values). The results are those of the
IEEE operations, so the tolerance is zero. Subnormal fields are compared with
the general kernels, on the lower rows as a level of its own: there the
oracle's halved sums round, and the operators' fused multiply-adds do not."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

cfmg = pytest.importorskip("cfmg")


def _fields(kind, sh, rng):
    i = np.arange(sh[0])[:, None, None]
    j = np.arange(sh[1])[None, :, None]
    if kind == "smooth":  # a field with nodal lines, and a rough right-hand side
        return np.sin(0.01 * i) * np.cos(0.013 * j), 1e-3 * rng.standard_normal(sh)
    if kind == "noise":
        return rng.standard_normal(sh), rng.standard_normal(sh)
    if kind == "ties":  # few bits, exponents close together: sums end exactly half way
        m = (1 << 52) + rng.integers(0, 4, sh) * (1 << rng.integers(0, 3, sh))
        return np.ldexp(m.astype(float), rng.integers(-56, -50, sh)) * rng.choice([-1, 1], sh), np.zeros(sh)
    if kind == "cancel":  # neighbours of opposite sign that differ in the last bits, and powers of two
        s = (-1.0) ** (i // 2 + j)
        x = s * (1.0 + np.ldexp(rng.integers(-3, 4, sh).astype(float), -52))
        return np.where((i + j) % 97 == 0, np.ldexp(s, rng.integers(-14, 1, sh)), x), rng.standard_normal(sh)
    if kind == "wide":  # up to, at and beyond the range that is held, strip by strip
        span = np.broadcast_to(np.array([0, 14, 15, 16, 17, 60])[(i // 60 + j // 16) % 6], sh)
        return rng.standard_normal(sh) * np.ldexp(1.0, -rng.integers(0, 1 << 30, sh) % (span + 1)), np.zeros(sh)
    if kind == "zeros":  # land of either sign
        x = rng.standard_normal(sh) * np.broadcast_to((i // 45 + j // 9) % 3 == 0, sh)
        b = rng.standard_normal(sh) * np.broadcast_to((i // 90 + j // 18) % 2 == 0, sh)
        x[(x == 0) & (rng.random(sh) < 0.9)] *= -1.0
        return np.where((i > 200) & (i < 300) & (x == 0), -0.0, x), np.where(rng.random(sh) < 0.5, b, -b)
    if kind == "small":  # subnormal and next to it
        return rng.standard_normal(sh) * np.ldexp(1.0, -1000 - (i // 40) * 4 + 0 * j), np.zeros(sh)
    x = rng.standard_normal(sh) * np.ldexp(1.0, 900)  # near the top, with values that are not finite
    x.ravel(order="K")[rng.choice(x.size, 200, replace=False)] = rng.choice([np.nan, np.inf, -np.inf, 1.7e308], 200)
    return x, rng.standard_normal(sh)


@pytest.mark.parametrize("nx,ny", [(514, 514), (536, 515), (541, 530), (1096, 260)])
def test_integer_sums(nx, ny):
    p = dict(nx=nx, ny=ny, nz=1, case="twod", location="vertices", operator="laplacian9", nlevels=2, omega=0.8)
    og = O.OracleGmg(p)
    mg = cfmg.get_gmg(cfmg.Param(**p, verbose=False))
    rng = np.random.default_rng(nx)
    sh = og.shape(1)
    i = np.arange(sh[0])[:, None, None]
    j = np.arange(sh[1])[None, :, None]
    m = np.asfortranarray(np.broadcast_to((i // 170 + j // 130) % 4 != 3, sh).astype(np.uint8))
    og.field(1, "msk")[...] = m
    og.setup_operators()
    mg.oper[1].msk = m
    cfmg.setup_operators(mg)
    half = cfmg.get_gmg(cfmg.Param(**dict(p, ny=130), verbose=False))  # too small for the integer form
    n2 = half.data[1].x.shape[1]
    half.oper[1].msk = np.asfortranarray(m[:, :n2])
    cfmg.setup_operators(half)
    assert (n2 - 6) * (sh[0] - 6) < 1 << 18 <= (sh[0] - 6) * (sh[1] - 6)

    def same(a, b, what):
        ok = (a.view(np.int64) == b.view(np.int64)) | (np.isnan(a) & np.isnan(b))
        assert ok.all(), (what, int((~ok).sum()))

    def put(f, a):
        a = np.asfortranarray(a)
        og.field(1, f)[...] = a
        mg.upload(1, f, a)
        half.upload(1, f, np.asfortranarray(a[:, :n2]))

    def check(f, what):
        a, b = og.field(1, f), mg.download(1, f)
        if what.startswith("small"):  # rows that the other level's upper edge does not reach
            a, b = half.download(1, f)[:, : n2 - 10], b[:, : n2 - 10]
        same(np.asfortranarray(a), np.asfortranarray(b), what + f)

    with np.errstate(all="ignore"):
        for kind in ("smooth", "noise", "ties", "cancel", "wide", "zeros", "small", "large"):
            x, b = _fields(kind, sh, rng)
            for f, a in (("x", x), ("y", x), ("b", b), ("r", b)):
                put(f, a)
            if kind != "large":  # a dry cell's residual is a select here and a product in the oracle
                og.residual(1)
                for g in (mg, half):
                    g.residual[1](g, 1)
                check("r", kind + " residual ")
            og.smooth(1, 1)
            for g in (mg, half):
                g.smoother[1](g, 1, 1)
            check("x", kind + " sweep ")
            check("y", kind + " sweep ")
    mg.close()
    half.close()
