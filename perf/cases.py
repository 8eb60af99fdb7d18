"""The work that users of this package have it do, as timed cases.

Every case goes through a public entry point: the numpy modules
(``parallelbeam.alg``, ``conebeam.alg``) on host arrays, or the device helpers
(``device``, ``autograd``) on CUDA tensors.  Sizes are those of the tests and
of ``bench.py`` or lie between them.  Inputs are analytic projections of
seeded ellipses (parallel beam, per slice) and ellipsoids (cone beam), scaled
to a largest line integral of 3, with Poisson noise.

``exact`` evaluates the same results in 64 bits with torch alone: a Siddon
trace of every ray, as a sparse matrix (parallel beam) or segment by segment
(cone beam), and the solvers' update rules on top of it.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "ccpi-reconstruction_b200"))
from ccpi.reconstruction import autograd  # noqa: E402
from ccpi.reconstruction import device as D  # noqa: E402
from ccpi.reconstruction.conebeam import alg as cone_alg  # noqa: E402
from ccpi.reconstruction.parallelbeam import alg as pb_alg  # noqa: E402

DEV = "cuda"
ALGS = {"cgls": 0, "sirt": 1, "mlem": 2, "cgls_tikhonov": 3, "cgls_TVreg": 4}


def listed():
    return [
        # the smallest call: one numpy CGLS call on a 16-row slab, as a
        # script runs it; plan set-up, copies and launches weigh most
        dict(name="pb host cgls small", kind="pb_host", alg="cgls", na=180, nv=16, nh=192,
             cor=96.25, log=True, iters=5),
        # an ordinary numpy SIRT call on transmission data, with a ragged
        # number of angles, columns and rows (50 rows pad to 52)
        dict(name="pb host sirt ragged", kind="pb_host", alg="sirt", na=361, nv=50, nh=385,
             cor=0.0, log=False, iters=10),
        # projector pair at two detector pixels per voxel, for a user's own
        # solver on device tensors
        dict(name="pb projectors binned", kind="pb_proj", na=300, nv=128, nh=512, res=2),
        # device MLEM on sizes that are multiples of nothing
        dict(name="pb mlem odd", kind="pb_solve", alg="mlem", n=255, nz=33, na=400, nh=383,
             iters=4),
        # many regularised problems of uneven sizes, solved together
        dict(name="pb tv batch", kind="pb_batch", alg="cgls_TVreg", count=16, wmax=384,
             sizes=4, iters=3),
        # the largest parallel-beam volume: a few SIRT iterations, weights
        # included
        dict(name="pb sirt large", kind="pb_solve", alg="sirt", n=768, nz=256, na=720, nh=768,
             iters=3),
        # the smallest cone call: projection and gradient of one small volume
        # on a default plan
        dict(name="cone grad small", kind="cone_grad", batch=1, n=64, na=90, nd=96, nv=96,
             scatter=False),
        # a training step's projector work: a batch of volumes forward, their
        # residuals backward
        dict(name="cone grad batch", kind="cone_grad", batch=8, n=256, na=360, nd=384, nv=384,
             scatter=True),
        # numpy cone SIRT on transmission data: centre search, then the
        # deterministic back projector
        dict(name="cone host sirt", kind="cone_host", alg="sirt", na=180, nh=192, nv=160,
             iters=5),
        # device CGLS-Tikhonov on an odd grid whose detector sees past the
        # far edge of the volume, default plan
        dict(name="cone tikhonov odd", kind="cone_solve", alg="cgls_tikhonov", n=151, na=240,
             nd=226, nv=300, scatter=False, iters=3),
        # one iteration of the largest cone solve, in a session kept over
        # many iterations
        dict(name="cone cgls large", kind="cone_session", n=512, na=720, nd=768, nv=768,
             scatter=True),
        # ring-artefact filter of a stack before it is reconstructed
        dict(name="ring filter", kind="ring", na=720, nh=768, nv=256, series=3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pb_host", "pb_proj", "pb_solve", "pb_solve", "pb_batch", "cone_grad",
                       "cone_grad", "cone_host", "cone_solve", "cone_session", "ring"])
    if kind == "pb_host":
        nh = _log_int(rng, 128, 512)
        return dict(kind=kind, alg=rng.choice(sorted(ALGS)), na=_log_int(rng, 90, 720),
                    nv=_log_int(rng, 8, 64), nh=nh,
                    cor=rng.choice([0.0, nh / 2 + round(rng.uniform(-8, 8), 2)]),
                    log=rng.random() < 0.5, iters=rng.randint(3, 5))
    if kind == "pb_proj":
        return dict(kind=kind, na=_log_int(rng, 90, 720), nv=4 * _log_int(rng, 4, 64),
                    nh=2 * _log_int(rng, 64, 384), res=rng.choice([1, 2, 4]))
    if kind == "pb_solve":
        n = _log_int(rng, 96, 640)
        nz = _log_int(rng, 8, 256)
        return dict(kind=kind, alg=rng.choice(["sirt", "mlem", "cgls"]), n=n,
                    nz=nz if rng.random() < 0.4 else (nz + 3) // 4 * 4,
                    na=_log_int(rng, 90, 720), nh=n + 2 * rng.randint(0, n // 4),
                    iters=rng.randint(2, 4))
    if kind == "pb_batch":
        return dict(kind=kind, alg=rng.choice(["cgls_tikhonov", "cgls_TVreg"]),
                    count=rng.randint(4, 16), wmax=rng.randint(96, 384),
                    sizes=rng.randint(1, 10 ** 6), iters=rng.randint(2, 3))
    if kind == "ring":
        return dict(kind=kind, na=_log_int(rng, 90, 900), nh=_log_int(rng, 96, 768),
                    nv=_log_int(rng, 8, 256), series=rng.randint(1, 3))
    big = {"cone_grad": 200, "cone_host": 192, "cone_solve": 200, "cone_session": 400}[kind]
    n = _log_int(rng, 48, big)
    nd = 2 * _log_int(rng, 0.6 * n, 0.8 * n)
    case = dict(kind=kind, na=_log_int(rng, 60, 360))
    if kind == "cone_host":
        case.update(alg=rng.choice(sorted(ALGS)), nh=2 * (n // 2), nv=4 * _log_int(rng, 8, n // 4),
                    iters=rng.randint(2, 4))
        return case
    case.update(n=n, nd=nd, nv=2 * int(nd / 2 * rng.choice([1.0, 1.0, 1.3])),
                scatter=rng.random() < 0.5)
    if kind == "cone_grad":
        case.update(batch=rng.randint(1, 4))
        if case["batch"] > 1:  # items of a batch start on 16-byte boundaries
            case.update(n=(n + 3) // 4 * 4)
    if kind == "cone_solve":
        case.update(alg=rng.choice(sorted(ALGS)), iters=rng.randint(2, 3))
    return case


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(DEV).manual_seed(seed)


def _u(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device=DEV, dtype=torch.float32)


def _poisson_log(p, i0, g):
    """Line integrals scaled to at most 3, as -log of noisy counts."""
    p = p * (3.0 / p.max())
    counts = torch.poisson(torch.exp(-p) * i0, generator=g).clamp_(min=1.0)
    return counts.div_(i0).log_().neg_()


def _parallel_data(seed, na, nv, nh, shift=0.0, count=10):
    """(na, nv, nh) noisy log projections of `count` ellipses per slice."""
    g = _gen(seed)
    w = nh / 1.5
    th = (torch.arange(na, device=DEV) * (math.pi / na)).view(na, 1, 1)
    h = (torch.arange(nh, device=DEV) - (nh - 1) / 2.0 - shift).view(1, 1, nh)
    out = torch.zeros(na, nv, nh, device=DEV)
    for _ in range(count):
        cx, cy = (_u(g, -0.4 * w, 0.4 * w, 1, nv, 1) for _ in range(2))
        a, b = (_u(g, 0.04 * w, 0.3 * w, 1, nv, 1) for _ in range(2))
        rot, rho = _u(g, 0.0, math.pi, 1, nv, 1), _u(g, 0.1, 1.0, 1, nv, 1)
        # the ray of column h runs along (cos, sin) at offset h along (-sin, cos)
        s = h - (cy * torch.cos(th) - cx * torch.sin(th))
        c, d = torch.cos(rot - th), torch.sin(rot - th)
        m2 = (a * d) ** 2 + (b * c) ** 2
        out += (2.0 * rho * a * b / m2) * (m2 - s * s).clamp_(min=0.0).sqrt_()
    return _poisson_log(out, 1.0e4, g)


def _cone_data(seed, na, nh, nv, hp, vp, s2o, o2d, size, count=8):
    """(na, nh, nv) noisy log projections of `count` ellipsoids."""
    g = _gen(seed)
    h = torch.as_tensor(hp, device=DEV, dtype=torch.float32).view(nh, 1)
    v = torch.as_tensor(vp, device=DEV, dtype=torch.float32).view(1, nv)
    length = torch.sqrt((s2o + o2d) ** 2 + h * h + v * v)
    out = torch.zeros(na, nh, nv, device=DEV)
    e = [(_u(g, -0.25 * size, 0.25 * size, 3).tolist(), _u(g, 0.03 * size, 0.22 * size, 3).tolist(),
          float(_u(g, 0.1, 1.0, 1))) for _ in range(count)]
    for a in range(na):
        c, s = math.cos(2 * math.pi * a / na), math.sin(2 * math.pi * a / na)
        p = (-s2o * c, -s2o * s, 0.0)
        d = (c * o2d - s * h - p[0], s * o2d + c * h - p[1], v)
        for cen, ax, rho in e:
            qa = (d[0] / ax[0]) ** 2 + (d[1] / ax[1]) ** 2 + (d[2] / ax[2]) ** 2
            w = [(p[i] - cen[i]) / ax[i] for i in range(3)]
            qb = (d[0] * (w[0] / ax[0]) + d[1] * (w[1] / ax[1])) + d[2] * (w[2] / ax[2])
            qc = w[0] ** 2 + w[1] ** 2 + w[2] ** 2 - 1.0
            out[a] += (qb * qb - qa * qc).clamp_(min=0.0).sqrt_().div_(qa).mul_(length).mul_(2 * rho)
    return _poisson_log(out, 5.0e3, g)


def _cone_geometry(case):
    """Voxel 1; source and detector at the distance and the detector of the
    width that the 512^3 benchmark has, relative to the volume."""
    n, nd, nv = case["n"], case["nd"], case["nv"]
    pix, s2o = 1.2 * n / nd, 500.0 / 512.0 * n
    hp = (np.arange(nd) - (nd - 1) / 2.0) * pix
    vp = (np.arange(nv) - (nv - 1) / 2.0) * pix
    return pix, s2o, hp, vp


def _cone_host_geometry(case):
    """Distances and pixel size of the cone demonstration phantom, for this
    detector; the mask radius is that of the fan."""
    s2s, s2d = 250.0, 987.0
    pix = 200.0 / case["nh"]
    hmax = pix * (case["nh"] - 1) / 2.0
    return s2s, s2d, pix, s2s * math.sin(math.atan(hmax / s2d))


def _batch_sizes(case):
    r = random.Random(case["sizes"])
    return [(r.randint(64, case["wmax"]), r.randint(8, 64), r.randint(90, 900),
             math.exp(r.uniform(math.log(1e-3), math.log(1e-1)))) for _ in range(case["count"])]


def _batch_problem(case, seed, i, size):
    w, nz, na, lam = size
    nh = round(1.5 * w)
    return _parallel_data(1000 * seed + i, na, nz, nh), np.arange(na) * (180.0 / na), lam


def _host_pixels(case, seed):
    shift = case["cor"] - case["nh"] / 2.0 if case["cor"] > 0 else 0.0
    return _parallel_data(seed, case["na"], case["nv"], case["nh"], shift)


def _ring_data(case, seed):
    """A log sinogram (na, nh, nv) with a fixed gain error per element."""
    p = _parallel_data(seed, case["na"], case["nv"], case["nh"]).transpose(1, 2)
    gain = 0.02 * torch.randn(case["nh"], case["nv"], generator=_gen(seed + 1), device=DEV)
    return (p + gain).contiguous()


def _volumes(case, seed):
    """(batch, n, n, n) smooth positive volumes with sharp inclusions."""
    g, n = _gen(seed), case["n"]
    c = torch.arange(n, device=DEV, dtype=torch.float32) + 0.5 - n / 2.0
    x, y, z = c.view(n, 1, 1), c.view(1, n, 1), c.view(1, 1, n)
    out = torch.zeros(case["batch"], n, n, n, device=DEV)
    for b in range(case["batch"]):
        for _ in range(6):
            cen, ax = _u(g, -0.25 * n, 0.25 * n, 3).tolist(), _u(g, 0.06 * n, 0.22 * n, 3).tolist()
            r = ((x - cen[0]) / ax[0]) ** 2 + ((y - cen[1]) / ax[1]) ** 2 + ((z - cen[2]) / ax[2]) ** 2
            out[b] += float(_u(g, 0.1, 1.0, 1)) * (r <= 1.0)
        out[b] += 0.05 * torch.rand(n, n, n, generator=g, device=DEV)
    return out


def prepare(case, seed):
    s, kind = dict(case), case["kind"]
    if kind == "pb_host":
        p = _host_pixels(case, seed)
        s["pixels"] = (p if case["log"] else torch.exp(-p)).cpu().numpy()
        s["angles"] = (np.arange(case["na"]) * (180.0 / case["na"])).astype(np.float32)
    elif kind == "cone_host":
        s2s, s2d, pix, _ = _cone_host_geometry(case)
        hp = (np.arange(case["nh"]) - (case["nh"] - 1) / 2.0) * pix
        vp = (np.arange(case["nv"]) - (case["nv"] - 1) / 2.0) * pix
        p = _cone_data(seed, case["na"], case["nh"], case["nv"], hp, vp, s2s, s2d - s2s, 50.0)
        s["pixels"] = torch.exp(-p).cpu().numpy()
        s["angles"] = (np.arange(case["na"]) * (360.0 / case["na"])).astype(np.float32)
    elif kind == "pb_proj":
        s["plan"], nvp, voff = D.parallel_api_plan(
            case["na"], case["nv"], case["nh"], np.arange(case["na"]) * (180.0 / case["na"]),
            0.0, case["res"])
        s["sino"] = D.pack_parallel(_parallel_data(seed, case["na"], case["nv"], case["nh"]), nvp,
                                    voff)
        s["vol"] = _u(_gen(seed + 1), 0.0, 1.0, *s["plan"].shape)
        s["fp"], s["bp"] = torch.empty_like(s["sino"]), torch.empty_like(s["vol"])
    elif kind == "pb_solve":
        s["plan"] = D.parallel_plan((case["n"], case["n"], case["nz"]), case["na"], case["nh"])
        s["sino"] = _parallel_data(seed, case["na"], case["nz"], case["nh"]).transpose(1, 2).contiguous()
        s["x"] = torch.empty(s["plan"].shape, device=DEV)
    elif kind == "pb_batch":
        s["plans"], s["sinos"], s["xs"], s["lam"] = [], [], [], []
        for i, size in enumerate(_batch_sizes(case)):
            p, deg, lam = _batch_problem(case, seed, i, size)
            plan, nvp, voff = D.parallel_api_plan(*p.shape, deg, 0.0, 1)
            s["plans"].append(plan)
            s["sinos"].append(D.pack_parallel(p, nvp, voff))
            s["xs"].append(torch.empty(plan.shape, device=DEV))
            s["lam"].append(lam)
    elif kind == "ring":
        s["sino"] = _ring_data(case, seed)
        s["out"] = torch.empty_like(s["sino"])
    else:
        pix, s2o, hp, vp = _cone_geometry(case)
        s["plan"] = D.cone_plan(case["n"], 1.0, case["na"], case["nd"], pix, s2o, s2o,
                                n_det_v=case["nv"])
        s["plan"].set_cone_backprojector(case["scatter"])
        if kind == "cone_grad":
            s["vol"] = _volumes(case, seed).requires_grad_(True)
            s["target"] = _u(_gen(seed + 1), 0.0, 1.0, case["batch"], *s["plan"].sino_shape)
        else:
            s["sino"] = _cone_data(seed, case["na"], case["nd"], case["nv"], hp, vp, s2o, s2o,
                                   float(case["n"]))
            s["x"] = torch.zeros(s["plan"].shape, device=DEV)
        if kind == "cone_session":
            s["session"] = D.Session(s["plan"], ALGS["cgls"], s["sino"], s["x"], 100000)
    return s


def run(s):
    kind = s["kind"]
    if kind == "pb_host":
        args = [s["pixels"], s["angles"], s["cor"], 1, s["iters"], 1]
        norms = np.zeros(s["iters"])
        if s["alg"] in ("cgls_tikhonov", "cgls_TVreg"):
            args += [0.01, norms]
        return getattr(pb_alg, s["alg"])(*args, s["log"])
    if kind == "cone_host":
        s2s, s2d, pix, radius = _cone_host_geometry(s)
        zero = np.zeros(s["na"], np.float32)
        args = [s["pixels"], s["angles"], zero, zero, 1, s2s, s2d, pix, pix, radius, False,
                np.zeros(3, np.float32), np.zeros(3, np.float32), s["iters"], 1]
        if s["alg"] in ("cgls_tikhonov", "cgls_TVreg"):
            args += [0.01, np.zeros(s["iters"])]
        return getattr(cone_alg, s["alg"])(*args, False)
    if kind == "pb_proj":
        return s["plan"].forward(s["vol"], s["fp"]), s["plan"].backward(s["sino"], s["bp"])
    if kind == "pb_batch":
        for x in s["xs"]:
            x.zero_()
        return D.solve_batched(s["plans"], ALGS[s["alg"]], s["sinos"], s["xs"], s["iters"],
                               s["lam"])
    if kind == "ring":
        s["out"].copy_(s["sino"])
        return D.ring_filter_aml(s["out"], 0.1, 0.01, s["series"])
    if kind == "cone_grad":
        s["vol"].grad = None
        proj = autograd.project(s["vol"], s["plan"])
        proj.backward(s["target"])
        return proj.detach(), s["vol"].grad
    if kind == "cone_session":
        s["session"].run(1)
        return s["x"]
    s["x"].zero_()
    return s["plan"].solve(ALGS[s["alg"]], s["sino"], s["x"], s["iters"], 0.01)


# ------------------------------------------------------------------- work
def work(case):
    """One float read or written per input and output element.  Operations: a
    parallel ray spends a multiply and an add per crossed voxel and row, a
    cone ray 8 (two slices, their weights and sums); a ray of unit pixels
    crosses 4/pi cells per voxel length on average.  An iteration projects
    once each way; set-up back-projects once (CGLS, MLEM) or does both
    (SIRT)."""
    kind = case["kind"]
    if kind == "ring":
        n = case["na"] * case["nh"] * case["nv"]
        terms = 2 * case["series"] - 1
        return {"bytes": 8.0 * n, "flops": 4.0 * terms * n + 2.0 * terms * case["nh"] ** 2 * case["nv"]}
    if kind == "pb_batch":
        b = f = 0.0
        for w, nz, na, _ in _batch_sizes(case):
            nh = round(1.5 * w)
            b += 4.0 * (na * nh * nz + nh * nh * nz)
            f += 2.0 * na * nh * nh * nz * 4 / math.pi * (2 * case["iters"] + 1)
        return {"bytes": b, "flops": f}
    if kind.startswith("pb"):
        na, nh = case["na"], case["nh"]
        nz = case.get("nz", case.get("nv"))
        n = case.get("n", nh / case.get("res", 1))
        vol, sino = n * n * nz / case.get("res", 1), na * nh * nz
        one = 2.0 * na * n * n * case.get("res", 1) * nz * 4 / math.pi
        if kind == "pb_proj":
            return {"bytes": 8.0 * (vol + sino), "flops": 2 * one}
    else:
        na, nd, nv = case["na"], case.get("nd", case.get("nh")), case["nv"]
        n = case.get("n", nd)
        nz = case.get("n", nv)
        vol, sino = n * n * nz, na * nd * nv
        # rays per voxel at the axis: the fan's detector pitch, demagnified
        rays = nd / (0.6 * n) if "n" in case else 1.0
        one = 8.0 * na * n * n * rays * nv * 4 / math.pi
        if kind == "cone_grad":
            return {"bytes": 8.0 * case["batch"] * (vol + sino), "flops": 2 * case["batch"] * one}
        if kind == "cone_session":
            return {"bytes": 4.0 * (2 * vol + sino), "flops": 2 * one}
    passes = 2 * case["iters"] + {"sirt": 2}.get(case["alg"], 1)
    return {"bytes": 4.0 * (vol + sino), "flops": passes * one}


# ------------------------------------------------------------------ exact
F64 = torch.float64
EPS = 1.1920929e-07


def _trace(px, py, qx, qy, ox, oy, size, nx, ny):
    """Siddon in the plane: rays from (px, py) along (qx, qy) on an nx x ny
    grid.  Returns the sorted alphas (rays, segments + 1) clipped to the grid
    and each segment's cell (-1 outside or empty)."""
    def planes(p, q, o, n):
        flat = q.abs() < EPS * torch.sqrt(qx * qx + qy * qy)
        a = (o + torch.arange(n + 1, device=DEV, dtype=F64) * size - p[:, None]) / \
            torch.where(flat, torch.ones_like(q), q)[:, None]
        lo = torch.where(flat, -torch.inf, torch.minimum(a[:, 0], a[:, -1]))
        hi = torch.where(flat, torch.inf, torch.maximum(a[:, 0], a[:, -1]))
        return torch.where(flat[:, None], torch.nan, a), lo, hi
    ax, xlo, xhi = planes(px, qx, ox, nx)
    ay, ylo, yhi = planes(py, qy, oy, ny)
    lo = torch.maximum(xlo, ylo)
    hi = torch.maximum(torch.minimum(xhi, yhi), lo)
    a = torch.cat([ax, ay], 1)
    a = torch.where(torch.isnan(a), lo[:, None], a)
    a = a.clamp(lo[:, None], hi[:, None]).sort(1).values
    mid = 0.5 * (a[:, 1:] + a[:, :-1])
    i = torch.floor((px[:, None] + mid * qx[:, None] - ox) / size).long()
    j = torch.floor((py[:, None] + mid * qy[:, None] - oy) / size).long()
    ok = (i >= 0) & (i < nx) & (j >= 0) & (j < ny) & (a[:, 1:] > a[:, :-1])
    return a, torch.where(ok, i * ny + j, -1)


class _Parallel:
    """A and its transpose as sparse matrices over (ray, voxel column)."""
    MOST = 6e8  # nonzeros

    def __init__(self, angles, h, n, size, nz, rows_per_slice):
        self.na, self.nh, self.n, self.nz, self.rows = len(angles), len(h), n, nz, rows_per_slice
        th = torch.as_tensor(angles, device=DEV, dtype=F64).repeat_interleave(len(h))
        hv = torch.as_tensor(h, device=DEV, dtype=F64).repeat(len(angles))
        c, s = torch.cos(th), torch.sin(th)
        o = -n * size / 2.0
        rays, cells, lens = [], [], []
        step = max(1, 2 ** 24 // n)
        for r in range(0, len(th), step):
            cc, ss, hh = c[r:r + step], s[r:r + step], hv[r:r + step]
            a, cell = _trace(-ss * hh, cc * hh, cc, ss, o, o, size, n, n)
            k = (cell >= 0).nonzero()
            rays.append(k[:, 0] + r)
            cells.append(cell[k[:, 0], k[:, 1]])
            lens.append((a[:, 1:] - a[:, :-1])[k[:, 0], k[:, 1]])
        rays, cells, lens = torch.cat(rays), torch.cat(cells), torch.cat(lens)
        shape = (self.na * self.nh, n * n)
        self.a = self._csr(rays, cells, lens, shape)
        order = torch.argsort(cells, stable=True)
        self.at = self._csr(cells[order], rays[order], lens[order], shape[::-1])

    @staticmethod
    def _csr(rows, cols, vals, shape):
        at = torch.zeros(shape[0] + 1, device=DEV, dtype=torch.long)
        at[1:] = torch.cumsum(torch.bincount(rows, minlength=shape[0]), 0)
        return torch.sparse_csr_tensor(at, cols, vals, shape)

    def fp(self, x):
        y = self.a @ x.reshape(self.n * self.n, self.nz)
        return y.repeat_interleave(self.rows, 1).reshape(self.na, self.nh, -1)

    def bp(self, y):
        y = y.reshape(self.na * self.nh, self.nz, self.rows).sum(2)
        return (self.at @ y.contiguous()).reshape(self.n, self.n, self.nz)


class _Cone:
    """Segment by segment: a ray's piece inside one voxel column crosses at
    most one slice plane for every row (true of these geometries)."""

    def __init__(self, angles, hp, vp, s2o, o2d, n):
        t = lambda x: torch.as_tensor(np.asarray(x), device=DEV, dtype=F64)  # noqa: E731
        self.angles, self.h, self.v, self.n, self.s2o, self.o2d = angles, t(hp), t(vp), n, s2o, o2d
        self.length = torch.sqrt((s2o + o2d) ** 2 + self.h[:, None] ** 2 + self.v[None] ** 2)

    def _pieces(self):
        """For every angle and group of columns: index of both slices' voxels
        and both weights, (columns, segments, rows) each."""
        n, o = self.n, -self.n / 2.0
        step = max(1, int(2 ** 25 // (2 * n * len(self.v))))
        for ia, a in enumerate(self.angles):
            c, s = math.cos(a), math.sin(a)
            for h0 in range(0, len(self.h), step):
                h = self.h[h0:h0 + step]
                px, py = torch.full_like(h, -self.s2o * c), torch.full_like(h, -self.s2o * s)
                al, cell = _trace(px, py, c * self.o2d - s * h - px, s * self.o2d + c * h - py, o, o,
                                  1.0, n, n)
                keep = (cell >= 0).sum(1).max()
                first = torch.argsort((cell < 0).byte(), dim=1, stable=True)[:, :keep]
                cell = cell.gather(1, first)[:, :, None]
                a0, a1 = al[:, :-1].gather(1, first)[:, :, None], al[:, 1:].gather(1, first)[:, :, None]
                k = torch.floor(a0 * self.v - o)
                up = self.v > 0
                cut = torch.minimum((k + up + o) / self.v, a1)
                kn = k + torch.where(up, 1, -1)
                base = cell * n
                ok = cell >= 0
                yield (ia, h0, h0 + len(h),
                       (base + k).long(), torch.where(ok & (k >= 0) & (k < n), cut - a0, 0.0),
                       (base + kn).long(), torch.where(ok & (kn >= 0) & (kn < n), a1 - cut, 0.0))

    def fp(self, x):
        flat, last = x.reshape(-1), x.numel() - 1
        out = torch.zeros(len(self.angles), len(self.h), len(self.v), device=DEV, dtype=F64)
        for ia, h0, h1, i0, w0, i1, w1 in self._pieces():
            out[ia, h0:h1] = (flat[i0.clamp_(0, last)] * w0 + flat[i1.clamp_(0, last)] * w1).sum(1)
        return out * self.length

    def bp(self, y):
        out = torch.zeros(self.n ** 3, device=DEV, dtype=F64)
        y = y * self.length
        for ia, h0, h1, i0, w0, i1, w1 in self._pieces():
            p = y[ia, h0:h1, None, :]
            out.index_add_(0, i0.clamp_(0, len(out) - 1).view(-1), (p * w0).view(-1))
            out.index_add_(0, i1.clamp_(0, len(out) - 1).view(-1), (p * w1).view(-1))
        return out.reshape(self.n, self.n, self.n)


def _up(x, d):
    """x at the next index along d, mirrored at the end."""
    return torch.cat([x.narrow(d, 1, x.shape[d] - 1), x.narrow(d, x.shape[d] - 2, 1)], d)


def _dn(x, d):
    return torch.cat([x.narrow(d, 1, 1), x.narrow(d, 0, x.shape[d] - 1)], d)


def _laplace(x):
    return 0.25 * (_up(x, 0) + _dn(x, 0) + _up(x, 1) + _dn(x, 1)) - x


def _tv(x):
    """Divergence of the gradient normalised with minmod cross terms."""
    f = [_up(x, d) - x for d in range(3)]
    b = [x - _dn(x, d) for d in range(3)]
    m = [(0.5 * (f[d].sign() + b[d].sign()) * torch.minimum(f[d].abs(), b[d].abs())) ** 2
         for d in range(3)]
    total = 0.0
    for d in range(3):
        q = f[d] / torch.sqrt(f[d] ** 2 + sum(m[e] for e in range(3) if e != d) + EPS)
        total = total + (q - _dn(q, d))
    return total


def _solve(op, alg, b, x, iters, lam, clamp=True):
    inv = lambda t: torch.where(t > 0, 1.0 / t, 0.0)  # noqa: E731
    lam = float(np.float32(lam))
    if alg == "sirt":
        r, c = inv(op.fp(torch.ones_like(x))), inv(op.bp(torch.ones_like(b)))
        for _ in range(iters):
            x = (x + c * op.bp(r * (b - op.fp(x)))).clamp(min=0.0)
        return x
    if alg == "mlem":
        x, w = torch.ones_like(x), inv(op.bp(torch.ones_like(b)))
        for _ in range(iters):
            p = op.fp(x)
            x = (x * w * op.bp(torch.where(p != 0, b / p, 0.0).clamp(min=0.0))).clamp(min=0.0)
        return x
    reg = {"cgls": None, "cgls_tikhonov": _laplace, "cgls_TVreg": _tv}[alg]
    r, d = b, op.bp(b)
    g, t = d.square().sum(), torch.zeros_like(x)
    for _ in range(iters):
        q = op.fp(d)
        den = q.square().sum()
        if reg:
            t = t + lam * reg(d)
            den = den + t.square().sum()
        al = g / den
        x, r = x + al * d, r - al * q
        if reg:
            x = x + lam * reg(x)
        s = op.bp(r)
        g, be = s.square().sum(), s.square().sum() / g
        d = s + be * d
    return x.clamp(min=0.0) if clamp else x


def _api_grid(na, nv, nh, cor, res):
    """Columns' positions, cells per side, padded rows and first data row of
    the grid that the numpy calls derive from a parallel-beam detector."""
    shift = cor - nh / 2.0 if cor > 0 else 0.0
    h = np.arange(nh) - (nh - 1) / 2.0 - shift
    n = -(-math.ceil(2 * max(abs(h[0]), abs(h[-1]))) // res)
    while -res * n / 2.0 >= h[0] or res * n / 2.0 <= h[-1]:
        n += 1
    rows = -(-(-(-nv // res)) // 4) * 4 * res
    return h, n, rows, (rows - nv) // 2


def _pad_rows(p, rows, first):
    """(na, nv, nh) -> (na, nh, rows) in 64 bits."""
    out = torch.zeros(p.shape[0], p.shape[2], rows, device=DEV, dtype=F64)
    out[:, :, first:first + p.shape[1]] = p.transpose(1, 2)
    return out


def exact(case, seed):
    kind, na = case["kind"], case["na"] if "na" in case else 0
    rad = lambda deg: math.pi * (np.float32(deg).astype(np.float64) / 180.0)  # noqa: E731
    if kind == "pb_host":
        h, n, rows, first = _api_grid(na, case["nv"], case["nh"], case["cor"], 1)
        if 1.3 * na * n * n > _Parallel.MOST:
            return None
        p = _host_pixels(case, seed)
        p = p if case["log"] else -torch.log(torch.exp(-p).double())
        op = _Parallel(rad(np.arange(na) * (180.0 / na)), h, n, 1.0, rows, 1)
        x = torch.zeros(n, n, rows, device=DEV, dtype=F64)
        return _solve(op, case["alg"], _pad_rows(p, rows, first), x, case["iters"], 0.01).cpu().numpy()
    if kind == "pb_proj":
        res = case["res"]
        h, n, rows, first = _api_grid(na, case["nv"], case["nh"], 0.0, res)
        if 1.3 * na * n * n * res > _Parallel.MOST:
            return None
        op = _Parallel(rad(np.arange(na) * (180.0 / na)), h, n, float(res), rows // res, res)
        vol = _u(_gen(seed + 1), 0.0, 1.0, n, n, rows // res).double()
        p = _parallel_data(seed, na, case["nv"], case["nh"])
        return op.fp(vol), op.bp(_pad_rows(p, rows, first))
    if kind == "pb_solve":
        n, nh = case["n"], case["nh"]
        if 1.3 * na * n * n > _Parallel.MOST:
            return None
        op = _Parallel(np.arange(na) * (math.pi / na), np.arange(nh) - (nh - 1) / 2.0, n, 1.0,
                       case["nz"], 1)
        b = _pad_rows(_parallel_data(seed, na, case["nz"], nh), case["nz"], 0)
        x = torch.zeros(n, n, case["nz"], device=DEV, dtype=F64)
        return _solve(op, case["alg"], b, x, case["iters"], 0.01)
    if kind == "pb_batch":
        sizes = _batch_sizes(case)
        if sum(1.3 * a * (1.5 * w) ** 2 for w, _, a, _ in sizes) > 2.5 * _Parallel.MOST:
            return None
        out = []
        for i, size in enumerate(sizes):
            p, deg, lam = _batch_problem(case, seed, i, size)
            h, n, rows, first = _api_grid(*p.shape, 0.0, 1)
            op = _Parallel(rad(deg), h, n, 1.0, rows, 1)
            x = torch.zeros(n, n, rows, device=DEV, dtype=F64)
            out.append(_solve(op, case["alg"], _pad_rows(p, rows, first), x, case["iters"], lam))
        return out
    if kind == "ring":
        return _exact_ring(case, _ring_data(case, seed).double())
    if kind == "cone_host":
        return None  # the centre search's choice is part of the result
    pix, s2o, hp, vp = _cone_geometry(case)
    passes = {"cone_grad": 2 * case.get("batch", 1), "cone_session": 3}.get(
        kind, 2 * case.get("iters", 0) + 2)
    if passes * na * case["nd"] * case["nv"] * 1.3 * case["n"] > 6e10:
        return None
    op = _Cone(np.arange(na) * (2 * math.pi / na), hp, vp, s2o, s2o, case["n"])
    if kind == "cone_grad":
        vol = _volumes(case, seed).double()
        y = _u(_gen(seed + 1), 0.0, 1.0, case["batch"], na, case["nd"], case["nv"]).double()
        return (torch.stack([op.fp(v) for v in vol]), torch.stack([op.bp(t) for t in y]))
    b = _cone_data(seed, na, case["nd"], case["nv"], hp, vp, s2o, s2o, float(case["n"])).double()
    x = torch.zeros(case["n"], case["n"], case["n"], device=DEV, dtype=F64)
    if kind == "cone_session":
        return _solve(op, "cgls", b, x, 1, 0.0, clamp=False)
    return _solve(op, case["alg"], b, x, case["iters"], 0.01)


def _exact_ring(case, p):
    """Each angular term's profile, smoothed along the columns, is taken off."""
    na, nh = case["na"], case["nh"]
    par_n, par_r = 0.1, 0.01
    a = torch.arange(na, device=DEV, dtype=F64)
    terms = [torch.ones_like(a)]
    for k in range(1, case["series"]):
        terms += [math.sqrt(2) * torch.sin(a * (k * math.pi / na)),
                  math.sqrt(2) * torch.cos(a * (k * math.pi / na))]
    al = par_n + par_r
    tau = 2.0 * math.asinh(math.sqrt(al) / 2.0)
    i = torch.arange(1, nh + 1, device=DEV, dtype=F64)
    lo, hi = torch.minimum(i[:, None], i[None]), torch.maximum(i[:, None], i[None])
    ex = lambda t: torch.exp(-tau * t)  # noqa: E731
    mat = ex(hi - lo) * (1 + ex(2 * nh - 2 * hi + 1)) * (1 + ex(2 * lo - 1)) / \
        (math.sqrt(al * (al + 4.0)) * (1.0 - math.exp(-tau * 2 * nh)))
    for t, w in enumerate(terms):
        res = torch.einsum("ahv,a->hv", p, w) / na
        d = par_n * float(((t + 2) // 2) ** 2) * res
        d[:-1] += res[:-1] - res[1:]
        d[1:] += res[1:] - res[:-1]
        p = p - w[:, None, None] * (mat @ d)
    return p
