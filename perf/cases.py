"""The work that is timed: calls a user of this package makes, through its public entry points.

A case is a dict of plain values; its ``kind`` names the call:

* ``gram``          ``XRayTransform2D.gram`` of one small slice: A^T A x, the operator of every CG step.
* ``project``, ``back_project``   ``XRayTransform2D`` forward and adjoint of a slice or a few slices.
* ``fbp``           ``XRayTransform2D.fbp``: filtered back projection of one sinogram.
* ``project3d``, ``back_project3d``   ``XRayTransform3D`` forward and adjoint; rotation about volume axis 0
  (``seq`` "X", a parallel-beam tomogram) or tilted about two axes (``seq`` "XY", laminography).
* ``tv_step``       D x, the L2,1 prox of it and D^T of that: the regulariser's part of a step-by-step solver.
* ``tv_prox``       ``IsotropicTVNorm`` / ``AnisotropicTVNorm`` prox of a noisy image: one PGM / APGM step.
* ``cg_block``      ``inverse.cg_block`` forward and backward of a batch: MoDL's data-consistency block in training.
* ``admm``          a whole ``optimize.ADMM`` TV solve from a sinogram.

Images are sums of random ellipses (ellipsoids); sinograms are their exact line integrals with 0.5 % noise, so inputs
come from the seed alone.
"""

from __future__ import annotations

import math
import random

import numpy as np
import torch

from scico_gb300 import functional, inverse, linop, loss
from scico_gb300.optimize import ADMM, LinearSubproblemSolver

CAP2D = 1.1e8  # pixel-view interactions of the largest drawn 2D case
CAP3D = 256**3 * 360  # voxel-view interactions of the largest drawn volume


def listed():
    return [
        # A thumbnail slice, as in interactive use and in the small scans of a batch: launches and host work count.
        {"name": "gram_128", "kind": "gram", "rows": 128, "cols": 128, "views": 90, "det": 183, "batch": 1},
        # The benchmark slice (512 x 512, 360 views, 725 bins), each direction of the projector by itself.
        {"name": "project_512", "kind": "project", "rows": 512, "cols": 512, "views": 360, "det": 725, "batch": 1},
        {"name": "back_project_512", "kind": "back_project", "rows": 512, "cols": 512, "views": 360, "det": 725,
         "batch": 1},
        # A quick reconstruction without iterations; an odd slice size, as cropped data has.
        {"name": "fbp_501", "kind": "fbp", "rows": 501, "cols": 501, "views": 360, "det": 709, "batch": 1},
        # The benchmark volume (256^3, 360 views about axis 0, 256 x 363 detector): the largest calls.
        {"name": "project_volume_256", "kind": "project3d", "n0": 256, "n1": 256, "n2": 256, "views": 360, "det0": 256,
         "det1": 363, "seq": "X"},
        {"name": "back_project_volume_256", "kind": "back_project3d", "n0": 256, "n1": 256, "n2": 256, "views": 360,
         "det0": 256, "det1": 363, "seq": "X"},
        # A tilted rotation axis, with the odd and unequal sides that such samples have.
        {"name": "project_tilted_128", "kind": "project3d", "n0": 97, "n1": 128, "n2": 111, "views": 60, "det0": 128,
         "det1": 181, "seq": "XY"},
        {"name": "back_project_tilted_128", "kind": "back_project3d", "n0": 97, "n1": 128, "n2": 111, "views": 60,
         "det0": 128, "det1": 181, "seq": "XY"},
        # The regulariser on a volume, operator by operator.
        {"name": "tv_step_volume_192", "kind": "tv_step", "n0": 192, "n1": 192, "n2": 192, "lam": 0.05},
        # The TV prox of an image in a proximal gradient step.
        {"name": "tv_prox_512", "kind": "tv_prox", "n0": 1, "n1": 512, "n2": 512, "lam": 0.05, "norm": "iso",
         "circular": False},
        # One unrolled block of the training benchmark (16 slices of 256 x 256, 180 views, lambda 0.1); six CG steps,
        # where the step sizes and their gradients are still determined in 32 bits.
        {"name": "cg_block_16x256", "kind": "cg_block", "rows": 256, "cols": 256, "views": 180, "det": 363, "batch": 16,
         "iters": 6, "lam": 0.1},
        # A whole iterative reconstruction of the benchmark slice: two warm-started CG steps an iteration, the penalty
        # scaled to the data term (A^T A grows with views times columns).
        {"name": "admm_512", "kind": "admm", "rows": 512, "cols": 512, "views": 360, "det": 725, "iters": 20,
         "cg_iters": 2, "rho": 1000.0, "lam": 2.5},
    ]


def _log(rng: random.Random, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _slice(rng, lo, hi, vlo, vhi, cap):
    """Sides, view count and a detector that holds the image's diagonal."""
    while True:
        rows = _log(rng, lo, hi)
        cols = rows if rng.random() < 0.5 else max(lo, min(hi, int(rows * rng.uniform(0.7, 1.4))))
        views = _log(rng, vlo, vhi)
        if rows * cols * views <= cap:
            return {"rows": rows, "cols": cols, "views": views,
                    "det": int(math.ceil(math.hypot(rows, cols))) + rng.choice([0, 1, 1, 2, 16])}


def draw(rng):
    kind = rng.choice(["gram", "project", "back_project", "fbp", "project3d", "back_project3d", "project_tilted",
                       "back_project_tilted", "tv_step", "tv_prox", "cg_block", "admm"])
    if kind == "gram":
        return {"kind": kind, **_slice(rng, 64, 256, 45, 180, CAP2D), "batch": 1}
    if kind in ("project", "back_project"):
        c = _slice(rng, 160, 768, 60, 720, CAP2D)
        most = int(CAP2D // (c["rows"] * c["cols"] * c["views"]))
        return {"kind": kind, **c, "batch": rng.choice([1, 1, min(most, rng.randint(1, 8))])}
    if kind == "fbp":
        return {"kind": kind, **_slice(rng, 160, 768, 60, 720, CAP2D), "batch": 1}
    if kind in ("project3d", "back_project3d"):
        while True:
            n = [_log(rng, 48, 256) for _ in range(3)]
            views = _log(rng, 45, 360)
            if n[0] * n[1] * n[2] * views <= CAP3D:
                break
        return {"kind": kind, "n0": n[0], "n1": n[1], "n2": n[2], "views": views, "det0": n[0],
                "det1": int(math.ceil(math.hypot(n[1], n[2]))) + rng.choice([0, 1, 8]), "seq": "X"}
    if kind in ("project_tilted", "back_project_tilted"):
        n = [rng.randint(40, 144) for _ in range(3)]
        return {"kind": kind.replace("_tilted", "3d"), "n0": n[0], "n1": n[1], "n2": n[2], "views": rng.randint(12, 72),
                "det0": int(n[0] * rng.uniform(1.0, 1.3)), "det1": int(math.ceil(math.hypot(n[1], n[2]))), "seq": "XY"}
    if kind == "tv_step":
        if rng.random() < 0.4:
            return {"kind": kind, "n0": 1, "n1": _log(rng, 128, 2048), "n2": _log(rng, 128, 2048),
                    "lam": rng.uniform(0.01, 0.1)}
        return {"kind": kind, "n0": _log(rng, 32, 256), "n1": _log(rng, 32, 256), "n2": _log(rng, 32, 256),
                "lam": rng.uniform(0.01, 0.1)}
    if kind == "tv_prox":
        three = rng.random() < 0.4
        n = [_log(rng, 24, 160) for _ in range(3)] if three else [1, _log(rng, 128, 1024), _log(rng, 128, 1024)]
        return {"kind": kind, "n0": n[0], "n1": n[1], "n2": n[2], "lam": rng.uniform(0.01, 0.1),
                "norm": rng.choice(["iso", "aniso"]), "circular": rng.random() < 0.4}
    if kind == "cg_block":
        c = _slice(rng, 64, 256, 45, 180, CAP2D)
        most = int(16 * 256 * 256 * 180 // (c["rows"] * c["cols"] * c["views"]))
        return {"kind": kind, **c, "batch": max(1, min(most, rng.randint(1, 16))), "iters": rng.randint(3, 6),
                "lam": round(math.exp(rng.uniform(math.log(0.05), math.log(0.15))), 4)}
    c = _slice(rng, 128, 512, 60, 360, 512 * 512 * 360)
    return {"kind": kind, **c, "iters": rng.randint(8, 20), "cg_iters": rng.randint(1, 2),
            "rho": round(c["views"] * c["cols"] / 184.0, 2), "lam": round(c["views"] * c["cols"] / 73600.0, 4)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

DEV = "cuda"


def _ellipses(rng: random.Random, count: int, nd: int):
    """Centres, inverse axes maps L (unit ball = |L (p - c)| <= 1) and values, positions in units of half a side."""
    out = []
    for _ in range(count):
        c = [rng.uniform(-0.55, 0.55) for _ in range(nd)]
        axes = [rng.uniform(0.05, 0.4) for _ in range(nd)]
        q, _ = np.linalg.qr(np.array([[rng.gauss(0, 1) for _ in range(nd)] for _ in range(nd)]))
        out.append((np.array(c), np.diag(1.0 / np.array(axes)) @ q, rng.uniform(0.1, 0.6)))
    return out


def _image(shape, ell):
    """The ellipses' sum at the pixel (voxel) centres."""
    nd = len(shape)
    grids = [((torch.arange(n, device=DEV) + 0.5) / n * 2 - 1).reshape([-1 if a == k else 1 for a in range(nd)])
             for k, n in enumerate(shape)]
    img = torch.zeros(shape, device=DEV)
    for c, L, val in ell:
        r2 = torch.zeros(shape, device=DEV)
        for row in L:
            r2 += sum(float(row[k]) * (grids[k] - float(c[k])) for k in range(nd)) ** 2
        img += val * (r2 <= 1.0)
    return img


def _line_integrals(points, direction, half, ell):
    """Integrals along p + t d (pixel units) of the ellipses; points (..., nd), |d| = 1, half the image's half sides."""
    out = torch.zeros(points.shape[:-1], device=DEV)
    for c, L, val in ell:
        Ls = torch.tensor(L / half[None, :], dtype=torch.float32, device=DEV)
        q = (points - torch.tensor(c * half, dtype=torch.float32, device=DEV)) @ Ls.T
        e = Ls @ torch.tensor(direction, dtype=torch.float32, device=DEV)
        qe, ee = q @ e, float(e @ e)
        disc = qe * qe - ee * ((q * q).sum(-1) - 1.0)
        out += (2.0 * val / ee) * disc.clamp(min=0.0).sqrt()
    return out


def _noisy(y, gen):
    return y + (0.005 * float(y.abs().max())) * torch.randn(y.shape, generator=gen, device=DEV)


def _angles(views):
    return np.linspace(0, np.pi, views, endpoint=False)


def _sinogram(case, ell):
    """Line integrals over the bins of XRayTransform2D's default geometry (pixel side sqrt(2)/2 of a bin)."""
    dx = math.sqrt(2) / 2
    half = np.array([case["rows"], case["cols"]]) / 2.0
    s = (torch.arange(case["det"], device=DEV) + 0.5 - case["det"] / 2) / dx  # pixels from the centre
    rows = []
    for a in _angles(case["views"]):
        u = np.array([math.cos(a), math.sin(a)])
        pts = s[:, None] * torch.tensor(u, dtype=torch.float32, device=DEV)
        rows.append(_line_integrals(pts, np.array([-u[1], u[0]]), half, ell) / dx)
    return torch.stack(rows)


def _matrices(case):
    views = case["views"]
    shape, det = (case["n0"], case["n1"], case["n2"]), (case["det0"], case["det1"])
    if case["seq"] == "X":
        angles = _angles(views)[:, None]
    else:
        angles = np.stack([_angles(views), np.full(views, np.pi / 12)], axis=1)
    return linop.XRayTransform3D.matrices_from_euler_angles(shape, det, case["seq"], angles)


def _projections(case, matrices, ell):
    half = np.array([case["n0"], case["n1"], case["n2"]]) / 2.0
    r, c = torch.meshgrid(torch.arange(case["det0"], device=DEV) + 0.5, torch.arange(case["det1"], device=DEV) + 0.5,
                          indexing="ij")
    out = []
    for m in matrices:
        inv = torch.tensor(np.linalg.pinv(m[:, :3]), dtype=torch.float32, device=DEV)
        rc = torch.stack([r, c], -1) - torch.tensor(m[:, 3], dtype=torch.float32, device=DEV)
        d = np.cross(m[0, :3], m[1, :3])
        pts = rc @ inv.T - torch.tensor(half, dtype=torch.float32, device=DEV)
        out.append(_line_integrals(pts, d / np.linalg.norm(d), half, ell))
    return torch.stack(out)


def _slice_op(case):
    return linop.XRayTransform2D((case["rows"], case["cols"]), _angles(case["views"]), det_count=case["det"])


def _side(case):
    return tuple(n for n in (case["n0"], case["n1"], case["n2"]) if n > 1)


def prepare(case, seed):
    rng = random.Random(seed)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind in ("gram", "project", "back_project", "fbp", "cg_block", "admm"):
        s["A"] = _slice_op(case)
        s["A"].geometry()  # the view table goes to the device when the operator is set up
        shape = (case["rows"], case["cols"])
        batch = case.get("batch", 1)
        if kind in ("gram", "project"):
            x = torch.stack([_image(shape, _ellipses(rng, 10, 2)) for _ in range(batch)])
            s["x"] = x[0].contiguous() if batch == 1 else x
        elif kind in ("back_project", "fbp", "admm"):
            y = torch.stack([_noisy(_sinogram(case, _ellipses(rng, 10, 2)), gen) for _ in range(batch)])
            s["y"] = y[0].contiguous() if batch == 1 else y
            if kind == "fbp":
                s["A"].fbp(s["y"])  # the operator keeps its detector mask from the first call on
            if kind == "admm":
                s["D"] = linop.FiniteDifference(shape, append=0)
        else:
            # the projector normalised by 1 / N, as the training scripts do
            s["H"] = (1.0 / max(shape)) * s["A"]
            x = torch.stack([_image(shape, _ellipses(rng, 10, 2)) for _ in range(batch)])
            # b = H^T y + lam z and the starting image z: a blurred, noisy version of the slice
            z = torch.nn.functional.avg_pool2d(x[:, None], 5, 1, 2)[:, 0]
            z = z + 0.02 * torch.randn(z.shape, generator=gen, device=DEV)
            blur = torch.nn.functional.avg_pool2d(x[:, None], 31, 1, 15)[:, 0]
            s["b"] = (0.6 * blur + case["lam"] * z).contiguous().requires_grad_()
            s["x0"] = z.contiguous().requires_grad_()
            s["lam"] = torch.tensor([case["lam"]], device=DEV, requires_grad=True)
            s["gx"] = (2.0 / x.numel()) * (z - x + 0.05 * torch.randn(z.shape, generator=gen, device=DEV))
    elif kind in ("project3d", "back_project3d"):
        m = _matrices(case)
        shape, det = (case["n0"], case["n1"], case["n2"]), (case["det0"], case["det1"])
        s["A"] = linop.XRayTransform3D(shape, m, det)
        s["A"].geometry()
        ell = _ellipses(rng, 10, 3)
        if kind == "project3d":
            s["x"] = _image(shape, ell)
        else:
            s["y"] = _noisy(_projections(case, m, ell), gen)
    else:
        shape = _side(case)
        x = _image(shape, _ellipses(rng, 10, len(shape)))
        s["x"] = x + 0.05 * torch.randn(shape, generator=gen, device=DEV)
        if kind == "tv_step":
            s["D"], s["g"] = linop.FiniteDifference(shape, append=0), functional.L21Norm()
        else:
            cls = functional.IsotropicTVNorm if case["norm"] == "iso" else functional.AnisotropicTVNorm
            s["g"] = cls(circular=case["circular"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "gram":
        return s["A"].gram(s["x"])
    if kind in ("project", "project3d"):
        return s["A"].project(s["x"])
    if kind in ("back_project", "back_project3d"):
        return s["A"].back_project(s["y"])
    if kind == "fbp":
        return s["A"].fbp(s["y"])
    if kind == "tv_step":
        z = s["g"].prox(s["D"](s["x"]), case["lam"])
        return [z, s["D"].adj(z)]
    if kind == "tv_prox":
        return s["g"].prox(s["x"], case["lam"])
    if kind == "cg_block":
        x = inverse.cg_block(s["H"], s["b"], s["lam"], s["x0"], maxiter=case["iters"])
        gb, gl, gx0 = torch.autograd.grad(x, (s["b"], s["lam"], s["x0"]), s["gx"])
        return [x.detach(), gb, gl, gx0]
    solver = ADMM(f=loss.SquaredL2Loss(y=s["y"], A=s["A"]), g_list=[case["lam"] * functional.L21Norm()],
                  C_list=[s["D"]], rho_list=[case["rho"]], maxiter=case["iters"],
                  subproblem_solver=LinearSubproblemSolver(cg_kwargs={"tol": 1e-6, "maxiter": case["cg_iters"]}))
    return solver.solve()


def work(case):
    kind = case["kind"]
    if kind in ("gram", "project", "back_project", "fbp", "cg_block", "admm"):
        img, sino = case["rows"] * case["cols"], case["views"] * case["det"]
        inter = img * case["views"]
        b = case.get("batch", 1)
        once = 8.0 * inter  # per pixel and view: Px, distance and weight (4), two multiply-adds (4)
        if kind == "gram":
            return {"bytes": 8.0 * img, "flops": 2 * once}
        if kind in ("project", "back_project"):
            return {"bytes": 4.0 * b * (img + sino), "flops": b * once}
        if kind == "fbp":
            return {"bytes": 4.0 * (img + sino), "flops": once + 1.0 * sino * case["det"]}
        if kind == "cg_block":  # forward: x0 and each step; backward: each step and x0
            return {"bytes": 4.0 * b * 6 * img, "flops": b * 2.0 * (case["iters"] + 1) * 2 * once}
        # A^T y, one pair per iteration and CG step
        return {"bytes": 4.0 * (img + sino), "flops": once * (1 + 2.0 * case["iters"] * (case["cg_iters"] + 1))}
    vol = case["n0"] * case["n1"] * case["n2"]
    if kind in ("project3d", "back_project3d"):
        per = 4.0 if case["seq"] == "X" else 24.0  # two taps; four taps and their weights
        return {"bytes": 4.0 * (vol + case["views"] * case["det0"] * case["det1"]),
                "flops": per * vol * case["views"]}
    nd = len(_side(case))
    if kind == "tv_step":
        return {"bytes": 4.0 * vol * (2 + nd), "flops": 8.0 * nd * vol}
    return {"bytes": 8.0 * vol, "flops": 14.0 * nd * vol}


# ---------------------------------------------------------------------------
# 64-bit results
# ---------------------------------------------------------------------------


class _Slice64:
    """XRayTransform2D's model in float64: pixel corner positions, boxcar of the projected pixel, two bins."""

    def __init__(self, case, scale=1.0):
        self.rows, self.cols, self.det, self.views = case["rows"], case["cols"], case["det"], case["views"]
        self.i = torch.arange(self.rows, device=DEV, dtype=torch.float64)[:, None]
        self.j = torch.arange(self.cols, device=DEV, dtype=torch.float64)[None, :]
        self.scale = scale

    def taps(self, a):
        dx = math.sqrt(2) / 2
        u0, u1 = math.cos(a), math.sin(a)
        p0 = -(self.rows * dx / 2) * u0 - (self.cols * dx / 2) * u1 + self.det / 2
        d0, d1 = dx * u0, dx * u1
        width = max(abs(d0), abs(d1))
        px = p0 + min(0.0, d0) + min(0.0, d1) + d0 * self.i + d1 * self.j
        k = px.floor()
        w = (1.0 - (px - k)).clamp(max=width) / width
        return k.long().reshape(-1) + 1, w.reshape(-1)  # bins shifted by one: 0 and det + 1 take what falls outside

    def fwd(self, x):
        b = x.shape[0]
        flat = x.reshape(b, -1)
        out = torch.zeros(b, self.views, self.det + 3, device=DEV, dtype=torch.float64)
        for v, a in enumerate(_angles(self.views)):
            k, w = self.taps(a)
            row = out[:, v]
            row.index_add_(1, k.clamp(0, self.det + 1), flat * w)
            row.index_add_(1, (k + 1).clamp(0, self.det + 1), flat * (1.0 - w))
        return self.scale * out[:, :, 1:self.det + 1]

    def adj(self, y):
        b = y.shape[0]
        out = torch.zeros(b, self.rows * self.cols, device=DEV, dtype=torch.float64)
        yp = torch.zeros(b, self.views, self.det + 3, device=DEV, dtype=torch.float64)
        yp[:, :, 1:self.det + 1] = y
        for v, a in enumerate(_angles(self.views)):
            k, w = self.taps(a)
            row = yp[:, v]
            out += row[:, k.clamp(0, self.det + 1)] * w + row[:, (k + 1).clamp(0, self.det + 1)] * (1.0 - w)
        return self.scale * out.reshape(b, self.rows, self.cols)

    def gram(self, x):
        return self.adj(self.fwd(x))


def _volume64(case, matrices, data):
    """XRayTransform3D with its float32 positions and weights (which decide the detector pixel: the model jumps where a
    position is a whole number) and 64-bit sums, for the volume or for the projections."""
    n, det = (case["n0"], case["n1"], case["n2"]), (case["det0"], case["det1"])
    m32 = np.asarray(matrices, dtype=np.float32)
    ax = [(torch.arange(k, device=DEV, dtype=torch.float32) + 0.5).reshape([-1 if a == q else 1 for a in range(3)])
          for q, k in enumerate(n)]
    forward = case["kind"] == "project3d"
    size = det[0] * det[1]
    d64 = data.double()
    out = torch.zeros((case["views"], size) if forward else n, device=DEV, dtype=torch.float64)
    for v in range(case["views"]):
        taps = []
        for r in range(2):
            m = [float(q) for q in m32[v, r]]
            px = ((m[0] * ax[0] + m[1] * ax[1]) + m[2] * ax[2]) + m[3]
            left = px - 0.25
            t = (left.ceil() - left).clamp(max=0.5)
            taps.append((left.floor().long(), t))
        for a in (0, 1):
            wa = taps[0][1] if a == 0 else 0.5 - taps[0][1]
            if not bool((wa != 0).any()):
                continue
            ia = taps[0][0] + a
            for b in (0, 1):
                wb = taps[1][1] if b == 0 else 0.5 - taps[1][1]
                ib = taps[1][0] + b
                ok = (ia >= 0) & (ia < det[0]) & (ib >= 0) & (ib < det[1])
                w = torch.where(ok, ((wa * wb) * 4.0).double(), 0.0)
                at = torch.where(ok, ia * det[1] + ib, 0).expand(n)
                if forward:
                    out[v].index_add_(0, at.reshape(-1), (w * d64).reshape(-1))
                else:
                    out += w * d64[v].reshape(-1)[at]
    return out.reshape(case["views"], *det) if forward else out


def _diff64(x):
    return torch.stack([torch.diff(x, dim=a, append=x.narrow(a, x.shape[a] - 1, 1)) for a in range(x.ndim)])


def _diff_adj64(d):
    out = torch.zeros_like(d[0])
    for a in range(d.shape[0]):
        n = out.shape[a]
        core = d[a].narrow(a, 0, n - 1)  # the last difference is zero times the repeated end sample
        out.narrow(a, 1, n - 1).add_(core)
        out.narrow(a, 0, n - 1).sub_(core)
    return out


def _shrink64(v, thr):
    length = (v * v).sum(0).sqrt()
    return v * torch.where(length > 0, (length - thr).clamp(min=0) / length.clamp(min=1e-300), 0.0)


def _tv_prox64(case, v):
    """1/K times the adjoint Haar transform of the transform of v with its highpass part shrunk."""
    nd = v.ndim
    K = 2 * nd
    thr = math.sqrt(2) * K * case["lam"]
    r = 1.0 / math.sqrt(2)
    x = v
    if not case["circular"]:
        for a in range(nd):
            x = torch.cat((x, x.narrow(a, x.shape[a] - 1, 1)), dim=a)
    lo = [r * (x + torch.roll(x, -1, a)) for a in range(nd)]
    hi = torch.stack([r * (torch.roll(x, -1, a) - x) for a in range(nd)])
    region = (slice(None),) + tuple(slice(0, n) for n in v.shape)
    part = hi[region]
    hi[region] = _shrink64(part, thr) if case["norm"] == "iso" else part.sign() * (part.abs() - thr).clamp(min=0)
    out = sum(r * (lo[a] + torch.roll(lo[a], 1, a)) + r * (torch.roll(hi[a], 1, a) - hi[a]) for a in range(nd))
    return out[tuple(slice(0, n) for n in v.shape)] / K


def _ramp64(y, det):
    n = np.arange(-(det - 1), det)
    h = np.where(n == 0, 0.25, np.where(n % 2 != 0, -1.0 / (np.pi**2 * np.where(n == 0, 1, n) ** 2.0), 0.0))
    # taps -(N-1)/2 .. N-1-(N-1)/2
    off = (det - 1) // 2
    h[(n < -off) | (n > det - 1 - off)] = 0.0
    k = torch.arange(det, device=DEV)
    T = torch.tensor(h, device=DEV)[(k[:, None] - k[None, :]) + det - 1]
    return y @ T.T


class _Gram64(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, A):
        ctx.A = A
        return A.gram(x)

    @staticmethod
    def backward(ctx, g):
        return ctx.A.gram(g), None


def _cg_block64(s, A):
    b = s["b"].detach().double().requires_grad_()
    x0 = s["x0"].detach().double().requires_grad_()
    lam = s["lam"].detach().double().requires_grad_()

    def op(u):
        return _Gram64.apply(u, A) + lam * u

    def dot(u, v):
        return (u * v).sum(dim=(1, 2), keepdim=True)

    x = x0
    r = b - op(x)
    p, num = r, dot(r, r)
    for _ in range(s["case"]["iters"]):
        Ap = op(p)
        alpha = num / dot(p, Ap)
        x, r = x + alpha * p, r - alpha * Ap
        new = dot(r, r)
        p, num = r + (new / num) * p, new
    gb, gl, gx0 = torch.autograd.grad(x, (b, lam, x0), s["gx"].double())
    return [x.detach(), gb, gl, gx0]


def _admm64(case, A, y):
    rho, lam = case["rho"], case["lam"]
    x = torch.zeros(case["rows"], case["cols"], device=DEV, dtype=torch.float64)
    z = _diff64(x)
    u = torch.zeros_like(z)
    aty = A.adj(y[None])[0]

    def op(p):
        return rho * _diff_adj64(_diff64(p)) + A.gram(p[None])[0]

    for _ in range(case["iters"]):
        b = aty + rho * _diff_adj64(z - u)
        r = b - op(x)
        p, num = r, float((r * r).sum())
        tol = (1e-6 * float(b.norm())) ** 2
        for _ in range(case["cg_iters"]):
            if num <= tol:
                break
            Ap = op(p)
            alpha = num / float((p * Ap).sum())
            x, r = x + alpha * p, r - alpha * Ap
            new = float((r * r).sum())
            p, num = r + (new / num) * p, new
        d = _diff64(x)
        z = _shrink64(d + u, lam / rho)
        u = u + d - z
    return x


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind in ("project3d", "back_project3d"):
        return _volume64(case, _matrices(case), s["x"] if kind == "project3d" else s["y"])
    if kind == "tv_step":
        z = _shrink64(_diff64(s["x"].double()), case["lam"])
        return [z, _diff_adj64(z)]
    if kind == "tv_prox":
        return _tv_prox64(case, s["x"].double())
    if kind == "cg_block":
        return _cg_block64(s, _Slice64(case, 1.0 / max(case["rows"], case["cols"])))
    A = _Slice64(case)
    if kind == "admm":
        return _admm64(case, A, s["y"].double())
    one = case["batch"] == 1
    d = (s["x"] if kind in ("gram", "project") else s["y"]).double()
    d = d[None] if one else d
    if kind == "fbp":
        # every pixel projects inside a detector that holds the diagonal: the mask is all ones
        out = (math.pi * 0.5 / case["views"]) * A.adj(_ramp64(d, case["det"]))
    else:
        out = {"gram": A.gram, "project": A.fwd, "back_project": A.adj}[kind](d)
    return out[0] if one else out
