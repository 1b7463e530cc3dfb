"""The measured work of this package: what its users have it do, through its public calls.

Every case is one pass of a user's program on a handle whose operators are set
up: a new right-hand side goes up, the call runs, the result comes back. The
right-hand sides and results live in device memory (``upload_ptr`` /
``download_ptr``), as they do in a model that runs on the GPU, except for the
adjoint, whose call takes and gives host arrays.

Kinds:
  solve    ``cfmg.solve`` from x = 0: the solution and the cycle count
  ops      the per-level function tables, as a program that writes its own
           cycle calls them, on coefficients that the program computed
  batch    ``Batch.solve`` of independent instances of uneven sizes
  adjoint  forward solve and ``cfmg.adjoint`` of the variable-coefficient
           operator, after a new kappa: the step of a parameter fit
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cfmultigrid.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import cfmg  # noqa: E402

NH = 3  # the reference's default halo
DEV = "cuda"


def _solve(nx, ny, nz, location, operator, cycle, sweeps, precision, mask, nlevels=0, topology="closed",
           tol=1e-10, omega=0.8):
    return dict(kind="solve", nx=nx, ny=ny, nz=nz, location=location, operator=operator, cycle=cycle,
                sweeps=sweeps, precision=precision, mask=mask, nlevels=nlevels, topology=topology, tol=tol,
                omega=omega)


def listed():
    return [
        # the smallest: one small elliptic solve inside a time step of a 2D
        # model, where launches and latency are what counts
        dict(name="solve-64-fp64", **_solve(64, 64, 1, "centers", "laplacian", "v", 2, "fp64", "disk")),
        # the plain method's configuration: 256^2 disk, 6 levels, FP64
        dict(name="solve-256-fp64", **_solve(256, 256, 1, "centers", "laplacian", "v", 2, "fp64", "disk", nlevels=6)),
        # a large drop-in solve in the default precision: vertex 9-point
        # F-cycle on a coastline of its own
        dict(name="solve-2048-fp64", **_solve(2048, 2048, 1, "vertices", "laplacian9", "f", 3,
                                              "fp64", "coast", nlevels=5)),
        # a 3D drop-in solve in the default precision, ragged extents
        dict(name="solve-3d-fp64", **_solve(208, 176, 112, "centers", "laplacian", "v", 2,
                                            "fp64", "basin", omega=0.84)),
        # the headline: 4096^2 vertex 9-point F-cycle, mixed precision, the
        # benchmark's coastline with a right-hand side of its own
        dict(name="solve-4096-mixed", **_solve(4096, 4096, 1, "vertices", "laplacian9", "f", 3,
                                               "mixed", "coast-1", nlevels=5)),
        # the large 3D ocean: coastline basin and bottom topography, V-cycle
        dict(name="solve-3d-mixed", **_solve(512, 512, 256, "centers", "laplacian", "v", 2,
                                             "mixed", "basin", nlevels=8, tol=1e-9)),
        # the 3D 19-point vertex operator in mixed precision
        dict(name="solve-3d19-mixed", **_solve(192, 192, 128, "vertices", "laplacian9", "v", 1,
                                               "mixed", "ball", tol=1e-9)),
        # an x-periodic channel with islands, ragged extents
        dict(name="channel-mixed", **_solve(1152, 608, 1, "centers", "laplacian", "v", 2,
                                            "mixed", "channel", topology="xperio")),
        # single operators of a ragged FP64 level, called through the tables
        dict(name="ops-fp64", kind="ops", nx=1930, ny=1415, mask="basin"),
        # a batch of independent uneven instances, sizes as the batched
        # configuration draws them
        dict(name="batch-128", kind="batch", count=128, lo=64, hi=1024),
        # a fit's step: new kappa, forward solve, adjoint
        dict(name="adjoint-2048", kind="adjoint", nx=2048, ny=2048, precision="mixed", tol=1e-12),
        # the same at an ordinary size in the default precision
        dict(name="adjoint-384-fp64", kind="adjoint", nx=384, ny=288, precision="fp64", tol=1e-12),
    ]


def _log_int(rng, lo, hi, step):
    return step * max(1, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step))


def draw(rng):
    kind = rng.choice(("2d-fp64", "2d-mixed", "coast", "3d-fp64", "3d-mixed", "3d19", "channel", "ops", "batch",
                       "adjoint"))
    sweeps = rng.choice((1, 2, 3))
    omega = rng.choice((0.8, 0.84, 0.9))
    if kind == "2d-fp64":  # a whole hierarchy; extents that coarsen through odd sizes
        n = _log_int(rng, 64, 1536, 4)
        location = rng.choice(("centers", "vertices"))
        return _solve(n, _log_int(rng, max(48, n // 2), n, 4), 1, location, rng.choice(("laplacian", "laplacian9")),
                      rng.choice("vf"), sweeps, "fp64", "basin" if location == "centers" else "disk", omega=omega)
    if kind == "2d-mixed":
        n = _log_int(rng, 256, 3072, 4)
        location = rng.choice(("centers", "vertices"))
        return _solve(n, _log_int(rng, n // 2, n, 4), 1, location, rng.choice(("laplacian", "laplacian9")),
                      rng.choice("vf"), sweeps, "mixed", "basin" if location == "centers" else "disk", omega=omega)
    if kind == "coast":
        n = _log_int(rng, 512, 2048, 16)
        return _solve(n, _log_int(rng, n // 2, n, 16), 1, "vertices", "laplacian9", "f", rng.choice((2, 3)),
                      rng.choice(("fp64", "mixed")), "coast", nlevels=5)
    if kind in ("3d-fp64", "3d-mixed"):
        n = _log_int(rng, 48, 160 if kind == "3d-fp64" else 320, 8)
        return _solve(n, _log_int(rng, max(48, n // 2), n, 8), _log_int(rng, 32, max(33, n // 2), 8), "centers",
                      "laplacian", "v", rng.choice((2, 3)), kind[3:], "basin", omega=rng.choice((0.8, 0.84)),
                      tol=1e-9)
    if kind == "3d19":
        n = _log_int(rng, 48, 176, 8)
        return _solve(n, n, _log_int(rng, 32, n, 8), "vertices", "laplacian9", "v", 1, "mixed", "ball",
                      tol=1e-9)
    if kind == "channel":
        return _solve(_log_int(rng, 128, 1152, 32), _log_int(rng, 96, 608, 8), 1, "centers", "laplacian", "v",
                      2, rng.choice(("mixed", "fp64")), "channel", topology="xperio")
    if kind == "ops":
        return dict(kind="ops", nx=_log_int(rng, 50, 1900, 1), ny=_log_int(rng, 50, 1400, 1), mask="basin")
    if kind == "batch":
        return dict(kind="batch", count=_log_int(rng, 16, 96, 1), lo=64, hi=rng.choice((512, 768, 1024)))
    n = _log_int(rng, 128, 1024, 16)
    return dict(kind="adjoint", nx=n, ny=_log_int(rng, n // 2, n, 16), precision=rng.choice(("mixed", "fp64")),
                tol=1e-12)


# ------------------------------------------------------------------ inputs
# Arrays are (tz, ty, tx) tensors in C order: the package's column-major
# (tx, ty, tz).
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed & 0x7FFFFFFF)


def _smooth(noise, sigma):
    """Periodic Gaussian smoothing of a 2D field."""
    ny, nx = noise.shape
    fy = torch.fft.fftfreq(ny, device=DEV, dtype=torch.float64)[:, None]
    fx = torch.fft.rfftfreq(nx, device=DEV, dtype=torch.float64)[None, :]
    damp = torch.exp(-2.0 * (math.pi * sigma) ** 2 * (fx * fx + fy * fy))
    return torch.fft.irfft2(torch.fft.rfft2(noise) * damp, s=(ny, nx))


def _centres(n):
    return (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) / n - 0.5


def _disk(nx, ny, radius):
    x, y = _centres(nx)[None, :], _centres(ny)[:, None]
    return x * x + y * y < radius * radius


def _basin(nx, ny, g):
    """A wavy-coast basin, connected by construction (star-shaped), with three round islands off each other and
    off the coast: the Neumann operator needs one connected wet region."""
    x, y = _centres(nx)[None, :], _centres(ny)[:, None]
    th, r = torch.atan2(y, x), torch.sqrt(x * x + y * y)
    a = torch.rand(6, generator=g, device=DEV, dtype=torch.float64)
    ph = 2 * math.pi * torch.rand(6, generator=g, device=DEV, dtype=torch.float64)
    coast = 0.42 + sum(0.05 / m * a[m - 1] * torch.cos(m * th + ph[m - 1]) for m in range(1, 7)) * 0.6
    wet = r < coast
    for k in range(3):
        c, s = math.cos(2.1 * k + 0.4), math.sin(2.1 * k + 0.4)
        wet = wet & ((x - 0.2 * c) ** 2 + (y - 0.2 * s) ** 2 > (0.02 + 0.05 * a[k]) ** 2)
    return wet


def _corners(wet):
    """Vertex (i, j) is wet iff the four cells around it are (interior sizes alike)."""
    w = torch.nn.functional.pad(wet.to(torch.uint8)[None, None], (1, 1, 1, 1))[0, 0]
    return (w[1:-1, 1:-1] & w[:-2, 1:-1] & w[1:-1, :-2] & w[:-2, :-2]).bool()


def _halo(wet, nz, threed):
    """(ny, nx) or (nz, ny, nx) wet cells into the level's array with halos."""
    if wet.dim() == 2:
        wet = wet[None].expand(nz, -1, -1)
    h = NH if threed else 0
    return torch.nn.functional.pad(wet.to(torch.uint8)[None], (NH, NH, NH, NH, h, h))[0].contiguous()


def _default(case):
    """The interior that the operators keep: every cell, or the vertices off the closed boundary."""
    nx, ny, nz = case["nx"], case["ny"], case.get("nz", 1)
    d = torch.ones((nz, ny, nx), dtype=torch.bool, device=DEV)
    if case.get("location", "centers") == "vertices":
        d[:, 0, :] = False
        d[:, :, 0] = False
    return d


def _wet(case, g):
    """Wet cells (nz, ny, nx) of a case's mask."""
    nx, ny, nz = case["nx"], case["ny"], case.get("nz", 1)
    kind = case["mask"]
    vert = case.get("location", "centers") == "vertices"
    if kind in ("coast", "coast-1"):
        # smoothed noise, 30 % land. "coast": sigma 64 cells, with which 5 levels converge for every seed tried up to
        # 2048^2. "coast-1": the benchmark's own coastline (noise of seed 1, sigma 32 cells, edges mirrored); with
        # other seeds the reference's F-cycle may diverge there.
        if kind == "coast":
            n = _smooth(torch.randn((ny, nx), generator=g, device=DEV, dtype=torch.float64), 64.0)
        else:
            n = torch.from_numpy(np.random.default_rng(1).standard_normal((nx, ny)).T.copy()).to(DEV)
            n = torch.cat([n[:, :128].flip(1), n, n[:, -128:].flip(1)], dim=1)
            n = torch.cat([n[:128].flip(0), n, n[-128:].flip(0)], dim=0)
            n = _smooth(n, 32.0)[128:-128, 128:-128].contiguous()
        wet = n > torch.sort(n.reshape(-1))[0][int(0.3 * n.numel())]
    elif kind == "disk":
        wet = _disk(nx, ny, 0.45)
    elif kind == "ball":
        x, y, z = _centres(nx)[None, None, :], _centres(ny)[None, :, None], _centres(nz)[:, None, None]
        return (x * x + y * y + z * z < 0.2) & _default(case)
    elif kind == "channel":  # a zonal channel with islands
        x, y = _centres(nx)[None, :], _centres(ny)[:, None]
        wet = torch.ones((ny, nx), dtype=torch.bool, device=DEV)
        a = torch.rand(4, generator=g, device=DEV, dtype=torch.float64)
        for k in range(4):
            cx, cy = -0.36 + 0.24 * k, 0.18 * (-1) ** k
            wet = wet & ((x - cx) ** 2 + (y - cy) ** 2 > (0.02 + 0.06 * a[k]) ** 2)
    else:
        wet = _basin(nx, ny, g)
    if nz > 1:  # bottom topography: a column is wet down to its depth
        u = 0.2 + 0.8 * torch.rand((ny, nx), generator=g, device=DEV, dtype=torch.float64)
        depth = nz * _smooth(u, 4.0)
        k = torch.arange(1, nz + 1, device=DEV, dtype=torch.float64)[:, None, None]
        return wet[None] & (k <= depth[None]) & _default(case)
    if vert:
        wet = _corners(wet)
    return wet[None] & _default(case)


def _noise_rhs(m, g):
    """N(0,1) on the wet cells of mask m (uint8, with halos), their mean removed."""
    b = torch.randn(m.shape, generator=g, device=DEV, dtype=torch.float64)
    b *= m
    b -= (b.sum() / m.sum(dtype=torch.float64)) * m
    return b


def _zero_all(mg):
    for lev in range(1, mg.nlevels + 1):
        for f in ("x", "y", "r", "b"):
            cfmg.set_to_zero(mg, lev, f)


def _inputs(case, seed):
    """(mask with halos, right-hand side) of a solve."""
    g = _gen(seed)
    m = _halo(_wet(case, g), case["nz"], case["nz"] > 1)
    return m, _noise_rhs(m, g)


# ----------------------------------------------------------------- prepare
def _prepare_solve(case, seed):
    threed = case["nz"] > 1
    m, b = _inputs(case, seed)
    p = cfmg.Param(nx=case["nx"], ny=case["ny"], nz=case["nz"], nh=NH, case="threed" if threed else "twod",
                   location=case["location"], operator=case["operator"], cycle=case["cycle"], npre=case["sweeps"],
                   npost=case["sweeps"], omega=case["omega"], nlevels=case["nlevels"], topology=case["topology"],
                   precision=case["precision"], residual_norm="l2", tol=case["tol"], maxite=100, verbose=False)
    mg = cfmg.get_gmg(p)
    torch.cuda.synchronize()
    mg.upload_ptr(1, "msk", m.data_ptr())
    cfmg.fill(mg, 1, "msk")
    cfmg.setup_operators(mg)
    _zero_all(mg)
    mg.synchronize()
    return {"kind": "solve", "mg": mg, "b": b, "x": torch.empty_like(b)}


def _run_solve(s):
    mg = s["mg"]
    mg.upload_ptr(1, "b", s["b"].data_ptr())
    cfmg.fill(mg, 1, "b")  # the periodic halo; nothing to do for a closed domain
    cfmg.set_to_zero(mg, 1, "x")
    _, nite = cfmg.solve(mg)
    mg.download_ptr(1, "x", s["x"].data_ptr())
    return {"x": s["x"], "nite": nite}


def _ops_inputs(case, seed):
    """x, b and the two finest levels' coefficients, as a program with its own setup has them: 5-point diag, its
    inverse, a coarse cell is wet where a child is, restriction mean over its wet children's count, prolongation
    weights 9-3-3-1 over 16."""
    g = _gen(seed)
    nx, ny = case["nx"], case["ny"]
    m = _halo(_wet(case, g), 1, False)
    x = torch.randn(m.shape, generator=g, device=DEV, dtype=torch.float64) * m
    b = _noise_rhs(m, g)
    f = m[0].double()
    nb = torch.zeros_like(f)
    nb[1:-1, 1:-1] = f[1:-1, :-2] + f[1:-1, 2:] + f[:-2, 1:-1] + f[2:, 1:-1]
    diag = nb * f
    idiag = torch.where(diag > 0, 1.0 / diag.clamp(min=1.0), torch.zeros_like(diag))
    cnx, cny = nx // 2, ny // 2
    kids = torch.zeros((cny + 2 * NH, cnx + 2 * NH), dtype=torch.float64, device=DEV)
    inner = f[NH:NH + 2 * cny, NH:NH + 2 * cnx].reshape(cny, 2, cnx, 2)
    kids[NH:-NH, NH:-NH] = inner.sum(dim=(1, 3))
    rcoef = torch.where(kids > 0, 4.0 / kids.clamp(min=1.0), torch.zeros_like(kids))
    pcoef = f / 16.0
    cx = torch.randn(kids.shape, generator=g, device=DEV, dtype=torch.float64) * (kids > 0)
    return dict(m=m, x=x, b=b, diag=diag, idiag=idiag, rcoef=rcoef, pcoef=pcoef, cx=cx)


def _col(t):
    """A (ty, tx) or (1, ty, tx) tensor as the host's column-major (tx, ty, 1) array."""
    return t.reshape(t.shape[-2], t.shape[-1]).cpu().numpy().T[:, :, None]


def _prepare_ops(case, seed):
    i = _ops_inputs(case, seed)
    p = cfmg.Param(nx=case["nx"], ny=case["ny"], nz=1, nh=NH, case="twod", location="centers", operator="laplacian",
                   cycle="v", npre=2, npost=2, omega=0.8, nlevels=2, verbose=False)
    mg = cfmg.get_gmg(p)
    mg.bind_level(1, diag=_col(i["diag"]), idiag=_col(i["idiag"]), Pcoef=_col(i["pcoef"]), msk=_col(i["m"]))
    mg.bind_level(2, Rcoef=_col(i["rcoef"]), msk=_col((i["rcoef"] > 0).to(torch.uint8)))
    _zero_all(mg)
    mg.synchronize()
    out = {k: torch.empty_like(i[v]) for k, v in (("x", "x"), ("r", "x"), ("cb", "cx"))}
    torch.cuda.synchronize()
    return {"kind": "ops", "mg": mg, "x": i["x"], "b": i["b"], "cx": i["cx"], "out": out}


def _run_ops(s):
    mg, out = s["mg"], s["out"]
    mg.upload_ptr(1, "b", s["b"].data_ptr())
    mg.upload_ptr(1, "x", s["x"].data_ptr())
    mg.upload_ptr(2, "x", s["cx"].data_ptr())
    mg.smoother[1](mg, 1, 2)
    mg.residual[1](mg, 1)
    mg.restriction[1](mg, 1, "r")
    mg.download_ptr(1, "r", out["r"].data_ptr())
    mg.download_ptr(2, "b", out["cb"].data_ptr())
    mg.prolongation[1](mg, 1)
    mg.smoother[1](mg, 1, 1)
    mg.download_ptr(1, "x", out["x"].data_ptr())
    return dict(out)


def _prepare_batch(case, seed):
    g = _gen(seed)
    # sides spread evenly over their logarithm, in no order (golden-ratio sequence)
    u = [(0.618033988749895 * (i + 1)) % 1.0 for i in range(case["count"])]
    sizes = [32 * max(2, round(case["lo"] * (case["hi"] / case["lo"]) ** v / 32)) for v in u]
    levels = [int(math.floor(math.log2(n / 8))) + 1 for n in sizes]
    p = cfmg.Param(nx=64, ny=64, nz=1, nh=NH, case="twod", location="centers", operator="laplacian", cycle="f",
                   npre=2, npost=2, omega=0.8, precision="mixed", residual_norm="l2", tol=1e-10, maxite=100,
                   verbose=False)
    bt = cfmg.Batch(p, sizes, sizes, levels)
    total = sum((n + 2 * NH) ** 2 for n in sizes)
    b = torch.empty(total, dtype=torch.float64, device=DEV)
    at, o = [], 0
    for i, n in enumerate(sizes):
        wet = _disk(n, n, 0.45) if i % 2 else _basin(n, n, g)
        m = _halo(wet[None], 1, False)
        k = m.numel()
        b[o:o + k] = _noise_rhs(m, g).reshape(-1)
        torch.cuda.synchronize()
        mg = bt.instance(i)
        mg.upload_ptr(1, "msk", m.data_ptr())
        cfmg.setup_operators(mg)
        _zero_all(mg)
        at.append(o)
        o += k
    bt.instance(0).synchronize()
    return {"kind": "batch", "batch": bt, "b": b, "x": torch.empty_like(b), "at": at}


def _run_batch(s):
    bt, b, x = s["batch"], s["b"].data_ptr(), s["x"].data_ptr()
    for i, o in enumerate(s["at"]):
        bt.instance(i).upload_ptr(1, "b", b + 8 * o)
    _, nite, _ = bt.solve()
    for i, o in enumerate(s["at"]):
        bt.instance(i).download_ptr(1, "x", x + 8 * o)
    return {"x": s["x"], "nite": nite}


def _prepare_adjoint(case, seed):
    g = _gen(seed)
    nx, ny = case["nx"], case["ny"]
    nlev = int(math.floor(math.log2(min(nx, ny) / 8))) + 1
    m = _halo(_disk(nx, ny, 0.45)[None], 1, False)
    f = _smooth(torch.randn(m.shape[1:], generator=g, device=DEV, dtype=torch.float64), 16.0)
    kappa = torch.exp(0.5 * f / f.std())[None].contiguous()
    b = _noise_rhs(m, g)
    cot = _noise_rhs(m, g)  # dL/dx of a misfit to noisy observations
    p = cfmg.Param(nx=nx, ny=ny, nz=1, nh=NH, case="twod", location="centers", operator="varcoef", cycle="v", npre=2,
                   npost=2, omega=0.8, nlevels=nlev, precision=case["precision"], residual_norm="l2",
                   tol=case["tol"], maxite=100, verbose=False)
    mg = cfmg.get_gmg(p)
    torch.cuda.synchronize()
    mg.upload_ptr(1, "msk", m.data_ptr())
    mg.synchronize()
    return {"kind": "adjoint", "mg": mg, "kappa": kappa, "b": b, "cot": np.asfortranarray(_col(cot)),
            "x": torch.empty_like(b)}


def _run_adjoint(s):
    mg = s["mg"]
    mg.upload_ptr(1, "kappa", s["kappa"].data_ptr())
    cfmg.setup_operators(mg)
    _zero_all(mg)
    mg.upload_ptr(1, "b", s["b"].data_ptr())
    _, nite = cfmg.solve(mg)
    mg.download_ptr(1, "x", s["x"].data_ptr())
    gb, gk = cfmg.adjoint(mg, s["cot"])
    return {"x": s["x"], "nite": nite, "grad_b": gb, "grad_kappa": gk}


_PREPARE = {"solve": _prepare_solve, "ops": _prepare_ops, "batch": _prepare_batch, "adjoint": _prepare_adjoint}
_RUN = {"solve": _run_solve, "ops": _run_ops, "batch": _run_batch, "adjoint": _run_adjoint}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


# -------------------------------------------------------------------- work
def _sweep_flops(operator, threed):
    return {"laplacian": 9 if threed else 7, "laplacian9": 22 if threed else 12, "varcoef": 11}[operator]


def _solve_flops(cells, threed, operator, cycle, sweeps, cycles):
    """Sweeps and one residual a level and cycle, the hierarchy's sum, and a norm; nominal cycle counts."""
    ratio = 1 / 8 if threed else 1 / 4
    levels = 1 / (1 - ratio) if cycle == "v" else 1 / (1 - ratio) ** 2
    return cells * cycles * ((4 * sweeps + 1) * _sweep_flops(operator, threed) + 8) * levels


def work(case):
    """Each input read once (b, mask, kappa), each output written once; the operations of the cycles that such a
    solve takes (about 10 in 2D, 30 on the 3D basins)."""
    k = case["kind"]
    if k == "batch":
        lo, hi, c = case["lo"], case["hi"], case["count"]
        cells = c * (hi * hi - lo * lo) / (2 * math.log(hi / lo))  # mean of a log-uniform side's square
        return {"bytes": 17 * cells, "flops": _solve_flops(cells, False, "laplacian", "f", 2, 10)}
    nz = case.get("nz", 1)
    cells = (case["nx"] + 2 * NH) * (case["ny"] + 2 * NH) * (nz + 2 * NH if nz > 1 else 1)
    if k == "ops":  # x, b, diag, idiag, mask, Pcoef, coarse x and Rcoef in; x, r, coarse b out
        return {"bytes": cells * (5 * 8 + 1 + 2 * 8 + 3 * 2), "flops": cells * (6 * 7 + 7 + 2 + 6)}
    if k == "adjoint":
        return {"bytes": cells * (5 * 8 + 8 + 1),
                "flops": 2 * _solve_flops(cells, False, "varcoef", "v", 2, 14) + 12 * cells}
    return {"bytes": 17 * cells,
            "flops": _solve_flops(cells, nz > 1, case["operator"], case["cycle"], case["sweeps"],
                                  30 if nz > 1 else 10)}


# ------------------------------------------------------------------- exact
def _nine(x):
    """faces / 2 + diagonals / 4 of a 2D field with halos, in its interior."""
    f = x[1:-1, :-2] + x[1:-1, 2:] + x[:-2, 1:-1] + x[2:, 1:-1]
    d = x[:-2, :-2] + x[:-2, 2:] + x[2:, :-2] + x[2:, 2:]
    return 0.5 * f + 0.25 * d


def _exact_vertices9(case, seed):
    """The masked 9-point Dirichlet problem faces/2 + diagonals/4 - 3 x = b, by conjugate gradients."""
    m, b = _inputs(case, seed)
    w = m[0].double()

    def a(v):
        out = 3.0 * v
        out[1:-1, 1:-1] -= _nine(v)
        return out.mul_(w)

    x = torch.zeros_like(w)
    r = -b[0] * w
    p = r.clone()
    rr = torch.sum(r * r)
    stop = 1e-13 ** 2 * float(rr)
    for it in range(20000):
        q = a(p)
        al = rr / torch.sum(p * q)
        x += al * p
        r -= al * q
        new = torch.sum(r * r)
        p = r + (new / rr) * p
        rr = new
        if it % 50 == 49 and float(rr) <= stop:
            break
    return {"x": x[None], "nite": None}


def _exact_ops(case, seed):
    i = _ops_inputs(case, seed)
    om = 0.8
    b, m, dg, w = i["b"][0], i["m"][0].double(), i["diag"], om * i["idiag"]
    cx, rc, pc = i["cx"], i["rcoef"], i["pcoef"]
    ty, tx = b.shape
    n = tx * ty

    def s4(v):  # over the linear range of whole rows, as the reference's 2D loops
        v = v.reshape(-1)
        c = slice(tx, n - tx)
        return v[tx - 1:n - tx - 1] + v[tx + 1:n - tx + 1] + v[:n - 2 * tx] + v[2 * tx:], c

    def sweep(v):
        s, c = s4(v)
        out = torch.zeros_like(v).reshape(-1)
        out[c] = (1 - om) * v.reshape(-1)[c] - w.reshape(-1)[c] * (b.reshape(-1)[c] - s)
        return out.reshape(ty, tx)

    x = i["x"][0]
    for _ in range(4):
        x = sweep(x)
    s, c = s4(x)
    r = torch.zeros_like(x).reshape(-1)
    r[c] = m.reshape(-1)[c] * (dg.reshape(-1)[c] * x.reshape(-1)[c] + b.reshape(-1)[c] - s)
    r = r.reshape(ty, tx)
    cny, cnx = rc.shape[0] - 2 * NH, rc.shape[1] - 2 * NH
    cb = torch.zeros_like(rc)
    kids = r[NH:NH + 2 * cny, NH:NH + 2 * cnx].reshape(cny, 2, cnx, 2)
    cb[NH:-NH, NH:-NH] = rc[NH:-NH, NH:-NH] * kids.sum(dim=(1, 3))
    # prolongation: parents cover (n + 1) // 2 cells a side
    px, py = (case["nx"] + 1) // 2, (case["ny"] + 1) // 2
    core = lambda dj, di: cx[NH + dj:NH + dj + py, NH + di:NH + di + px]  # noqa: E731
    x = x.clone()
    for dj in (0, 1):
        for di in (0, 1):
            a, e = 2 * dj - 1, 2 * di - 1
            v = 3 * (core(0, e) + core(a, 0)) + core(a, e) + 9 * core(0, 0)
            rows = slice(NH + dj, NH + dj + 2 * py, 2)
            cols = slice(NH + di, NH + di + 2 * px, 2)
            x[rows, cols] += pc[rows, cols] * v
    for _ in range(2):
        x = sweep(x)
    return {"x": x[None], "r": r[None], "cb": cb}


def exact(case, seed):
    """The cell-centred solves have no value here: their operator's solutions differ by a constant, which the cycle
    picks. The same goes for the batch and the adjoint, whose forward solution and gradients carry it."""
    if case["kind"] == "ops":
        return _exact_ops(case, seed)
    if (case["kind"] == "solve" and case["nz"] == 1 and case["location"] == "vertices" and
            case["operator"] == "laplacian9"):
        return _exact_vertices9(case, seed)
    return None
