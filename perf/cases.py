"""The workloads whose speed is tracked: the calls that users of this package make, through its
public entry points, from a toy geometry to the clinical one.

A case is a dict of plain values.  ``op`` names the call:

  fp          forward projection of a batch of slices
  fp_grad     a data-fidelity step: FP of the image, and the gradient of
              0.5 |FP(x) - y|^2 through autograd (the exact adjoint)
  bp_grad     the unweighted backprojection layer, forward and backward
  fbp         filtered backprojection of a batch of sinograms
  fbp_grad    the FBP layer, forward and backward
  driver      the raw-file driver's step on host arrays: FP of slices, FBP of the sinograms
  fp_cone     cone-beam forward projection of a volume
  fdk         cone-beam FDK reconstruction
  fdk_grad    the FDK layer, forward and backward
  uneven      one uneven batch: FP, FBP and FBP adjoint of slices of different geometries, BF16

Sizes: ``n`` image edge, ``views``, ``cols`` channels, ``batch`` slices or volumes; ``rows``
detector rows and ``nz`` slices of the cone-beam calls; ``shift`` the detector's quarter-channel
offset; ``window`` 0 Ram-Lak, 1 Shepp-Logan; ``short`` a Parker-weighted short scan; ``cosine``
the Feldkamp cosine pre-weights.  The field of view is 358.4 mm wide and the fan 888 mm at the
detector whatever the sampling (the clinical geometry is 512 pixels of 0.7 mm and 888 channels).

``exact`` restates every operator in float64 torch: the ray-marched projector as a sum of
``grid_sample`` values, the pixel-driven backprojectors as gathers, the filter as a product with
its Toeplitz matrix, and the gradients as their transposes.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

import fanbeamctrecon_tensorflowop_gb300 as ct
from fanbeamctrecon_tensorflowop_gb300 import utils
from fanbeamctrecon_tensorflowop_gb300.batch import UnevenBatch

SID, SDD = 541.0, 949.0
FOV_MM, FAN_MM = 358.4, 888.0
PI_F = np.float32(3.14159265359)
DEV = "cuda"


def listed():
    base = {"window": 0, "shift": 0.0, "short": False, "cosine": False}

    def case(name, op, n, views, cols, batch, **more):
        return {"name": name, "op": op, "n": n, "views": views, "cols": cols, "batch": batch,
                **base, **more}

    return [
        # a notebook or a unit test: one toy slice, where a call's latency is its time
        case("fp_toy_1", "fp", 64, 90, 96, 1),
        # simulating a scan: a batch of clinical slices at once
        case("fp_clinical_32", "fp", 512, 984, 888, 32),
        # iterative reconstruction of one clinical slice: a gradient step
        case("fp_grad_clinical_1", "fp_grad", 512, 984, 888, 1),
        # training with a physics layer: a few slices of an odd geometry per step
        case("fp_grad_odd_5", "fp_grad", 383, 719, 733, 5, shift=0.25),
        # a learned primal-dual style block: BP layer on a ragged batch of clinical slices
        case("bp_grad_clinical_13", "bp_grad", 512, 984, 888, 13),
        # reconstructing a stack of clinical slices with the smooth window
        case("fbp_clinical_16", "fbp", 512, 984, 888, 16, window=1),
        # training a dual-domain network on short scans: FBP layer at reduced size
        case("fbp_grad_short_3", "fbp_grad", 256, 400, 512, 3, short=True, cosine=True),
        # the raw-file driver on one slice: host arrays in and out
        case("driver_slice_1", "driver", 512, 984, 888, 1),
        # simulating a cone-beam scan of a small volume
        case("fp_cone_256", "fp_cone", 256, 492, 512, 1, rows=32, nz=32),
        # reconstructing a clinical cone-beam volume, with Feldkamp's weights
        case("fdk_clinical", "fdk", 512, 984, 888, 1, rows=64, nz=64, cosine=True),
        # training on cone-beam volumes: the FDK layer at reduced size
        case("fdk_grad_256", "fdk_grad", 256, 360, 512, 1, rows=32, nz=32),
        # a loader's batch of scans from different protocols, each its own geometry
        case("uneven_24", "uneven", 512, 984, 888, 24),
    ]


def draw(rng):
    def logint(lo, hi):
        return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))

    op = rng.choice(["fp", "fp", "fp_grad", "fp_grad", "bp_grad", "fbp", "fbp", "fbp_grad",
                     "driver", "fp_cone", "fdk", "fdk_grad", "uneven"])
    n = logint(64, 512)
    scale = n / 512
    views = max(60, min(984, round(984 * scale * rng.uniform(0.7, 1.4))))
    cols = max(96, min(888, round(888 * scale * rng.uniform(0.7, 1.4))))
    if rng.random() < 0.5:  # channel counts of real detectors are multiples of 4 or more
        cols -= cols % 8
    c = {"op": op, "n": n, "views": views, "cols": cols, "batch": logint(1, 32),
         "window": rng.choice([0, 1]), "shift": rng.choice([0.0, 0.0, 0.25]),
         "short": False, "cosine": False}
    if op.endswith("_grad"):
        c["batch"] = logint(1, 16)
    if op in ("fbp", "fbp_grad"):
        c["short"] = rng.random() < 0.3
        c["cosine"] = rng.random() < 0.3
    elif op == "driver":
        c["batch"] = logint(1, 8)
        c["window"] = 0
    elif op == "uneven":
        c["batch"] = logint(3, 24)
    elif op in ("fp_cone", "fdk", "fdk_grad"):
        if op != "fdk":
            c["n"] = n = min(n, 300)
            c["views"], c["cols"] = min(views, 500), min(cols, 520)
        c["batch"] = rng.choice([1, 1, 2]) if n <= 256 else 1
        c["rows"], c["nz"] = logint(8, 40), logint(8, 40)
        c["cosine"] = rng.random() < 0.5
        c["shift"] = 0.0
    return c


# ---- geometry: the 16-float parameter vector of the operators and its float32 decoding ----------


def _param(c, n=None, views=None, cols=None):
    n, views, cols = n or c["n"], views or c["views"], cols or c["cols"]
    dcol = FAN_MM / cols / SDD
    full = 2.0 * math.pi
    if c["short"]:
        full = (math.pi + 2.0 * (cols * dcol / 2.0 + c["shift"] * dcol)) * views / (views - 1)
    p = np.arange(16, dtype=np.float32)
    p[:13] = [SDD, SID, views, math.degrees(full), cols, n, n, FOV_MM / 2.0, math.degrees(dcol),
              c["shift"], math.degrees(-cols * dcol / 2.0), 1, 0.0]
    rows = c.get("rows", 1)
    if rows > 1:  # rows of 1 mm at 64 rows, slices of 0.625 mm at 64 slices
        p[13:] = [-32.0, 64.0 / rows, 40.0 / c["nz"]]
    return p, (np.arange(views) * (full / views)).astype(np.float32)


class _Geom:
    """The operators' float32 decoding of the parameter vector, as Python floats."""

    def __init__(self, p, angles):
        f = np.float32
        self.D, self.R = float(p[0]), float(p[1])
        self.V, self.C, self.nx = int(p[2]), int(p[4]), int(p[5])
        self.dang = float(f(f(f(p[3]) / f(self.V)) * PI_F) / f(180))
        self.rfov, self.shift = float(p[7]), float(p[9])
        dx = f(f(2) * f(p[7])) / f(self.nx)
        self.dx, self.xmin = float(dx), float(f(-0.5) * f(self.nx) * dx)
        self.dcol = float(f(p[8]) * PI_F / f(180))
        self.left = float(f(p[10]) * PI_F / f(180))
        self.bottom, self.drow, self.dz = float(p[13]), float(p[14]), float(p[15])
        self.beta = torch.tensor(angles.astype(np.float64), device=DEV)

    # -- rays of one view: start, step (texture pixels), samples, and per channel its fan geometry
    def rays(self, v):
        i = torch.arange(self.C, device=DEV, dtype=torch.float64)
        gam = self.left + (i + 0.5) * self.dcol
        th = self.beta[v] + gam
        src, fov = self.R / self.dx, self.rfov / self.dx
        dist = src * torch.sin(gam)
        h = (fov * fov - dist * dist).clamp(min=0)
        x, sn, cs = torch.sqrt(h), torch.sin(th), torch.cos(th)
        n = torch.floor(2.0 * x / 0.125)
        ax, ay = -x * cs + dist * sn, -x * sn - dist * cs
        bx, by = x * cs + dist * sn, x * sn - dist * cs
        m = n.clamp(min=1)
        s0 = self.dx * (src * torch.cos(gam) + x)
        return ax + fov, ay + fov, (bx - ax) / m, (by - ay) / m, n, s0, -2.0 * self.dx * x / m

    # -- pixels inside the field of view: flat index, x, y
    def pixels(self):
        t = self.xmin + self.dx * (torch.arange(self.nx, device=DEV, dtype=torch.float64) + 0.5)
        y, x = torch.meshgrid(t, t, indexing="ij")
        at = torch.nonzero((x * x + y * y <= self.rfov * self.rfov).reshape(-1))[:, 0]
        return at, x.reshape(-1)[at], y.reshape(-1)[at]

    # -- columns of the pixels (x, y) in view v: the two clamped taps, the fraction, 1/(U^2+t^2), U
    def columns(self, v, x, y):
        c, s = -torch.cos(self.beta[v]), -torch.sin(self.beta[v])
        U, t = self.R + x * c + y * s, -x * s + y * c
        col = (torch.atan(t / U) - self.left) / self.dcol + self.shift
        ok = (col > 0) & (col < self.C)
        b = torch.floor(col - 0.5)
        i0, i1 = b.long().clamp(0, self.C - 1), (b.long() + 1).clamp(0, self.C - 1)
        return i0, i1, col - 0.5 - b, torch.where(ok, 1.0 / (U * U + t * t), 0.0), ok.double(), U

    def toeplitz(self, window):
        n = torch.arange(-(self.C - 1), self.C, device=DEV, dtype=torch.float64)
        pi, s2 = float(PI_F), torch.sin(n * self.dcol) ** 2
        if window:
            h = n * n / (pi * pi * s2 * (1.0 - 4.0 * n * n))
            h0 = 1.0 / (pi * pi * self.dcol ** 2)
        else:
            h = torch.where(n % 2 != 0, -0.5 / (pi * pi * s2), torch.zeros_like(n))
            h0 = 0.125 / self.dcol ** 2
        h[self.C - 1] = h0
        i = torch.arange(self.C, device=DEV)
        return (h * (self.R * self.dang * self.dcol))[i[:, None] - i[None, :] + self.C - 1]

    def preweights(self, c):
        """[V, rows, C] weights ahead of the filter, or None."""
        i = torch.arange(self.C, device=DEV, dtype=torch.float64)
        gam = self.left + (i + 0.5 - self.shift) * self.dcol
        w = None
        if c["short"]:
            G = float(gam.abs().max()) + 0.5 * self.dcol
            beta = (self.beta - self.beta[0])[:, None]

            def step(u):
                return torch.sin(0.5 * math.pi * u.clamp(0, 1)) ** 2

            w = 2.0 * step(beta / (2 * (G - gam))) * step((math.pi + 2 * G - beta) / (2 * (G + gam)))
            w = torch.where(beta <= math.pi + 2 * G, w, 0.0)[:, None, :]
        if c["cosine"]:
            rows = c.get("rows", 1)
            cw = torch.cos(gam)[None, None, :]
            if rows > 1:
                h = self.bottom + (torch.arange(rows, device=DEV, dtype=torch.float64) + 0.5) * self.drow
                cw = cw / torch.sqrt(1.0 + (h / self.D) ** 2)[None, :, None]
            w = cw if w is None else w * cw
        return w


# ---- inputs ----------------------------------------------------------------------------------


def _ellipsoids(g, c, gen, batch):
    """[batch, 9, 7]: centre x y z, semi-axes, density (1/mm) of a body with inserts."""
    u = torch.rand((batch, 9, 7), generator=gen, device=DEV, dtype=torch.float64)
    e = torch.empty_like(u)
    r, phi = 0.65 * g.rfov * torch.sqrt(u[..., 0]), 2 * math.pi * u[..., 1]
    half = 0.5 * g.dz * c.get("nz", 1)
    e[..., 0], e[..., 1], e[..., 2] = r * torch.cos(phi), r * torch.sin(phi), half * (u[..., 2] - 0.5)
    e[..., 3:5] = g.rfov * (0.05 + 0.25 * u[..., 3:5])
    e[..., 5] = half * (0.3 + 0.9 * u[..., 5])
    e[..., 6] = -0.01 + 0.03 * u[..., 6]
    e[:, 0, :2], e[:, 0, 3:5], e[:, 0, 5], e[:, 0, 6] = 0.0, 0.88 * g.rfov, 1.6 * half, 0.019
    return e


def _image(g, c, gen, batch):
    """Attenuation images (or volumes) of the bodies, with a little texture."""
    e = _ellipsoids(g, c, gen, batch)
    t = g.xmin + g.dx * (torch.arange(g.nx, device=DEV, dtype=torch.float64) + 0.5)
    nz = c.get("nz", 0)
    z = g.dz * (torch.arange(max(nz, 1), device=DEV, dtype=torch.float64) + 0.5 - 0.5 * max(nz, 1))
    out = torch.zeros((batch, max(nz, 1), g.nx, g.nx), device=DEV)
    for k in range(e.shape[1]):
        q = e[:, k, :, None]
        X, Y = ((t - q[:, 0]) / q[:, 3]) ** 2, ((t - q[:, 1]) / q[:, 4]) ** 2
        Z = ((z - q[:, 2]) / q[:, 5]) ** 2 if nz else torch.zeros((batch, 1), device=DEV).double()
        d = X[:, None, None, :] + Y[:, None, :, None] + Z[:, :, None, None]
        out += (e[:, k, 6, None, None, None] * (d <= 1.0)).float()
    out += 2e-4 * torch.randn(out.shape, generator=gen, device=DEV) * (out != 0)
    return out if nz else out[:, 0]


def _sinogram(g, c, gen, batch):
    """Noisy analytic projections of the bodies: [B, V, C], or [B, V, rows, C]."""
    e = _ellipsoids(g, c, gen, batch)
    rows = c.get("rows", 1)
    i = torch.arange(g.C, device=DEV, dtype=torch.float64)
    gam = g.left + (i + 0.5) * g.dcol
    th = g.beta[:, None] + gam
    h = torch.zeros(1, device=DEV, dtype=torch.float64)
    if rows > 1:
        h = g.bottom + (torch.arange(rows, device=DEV, dtype=torch.float64) + 0.5) * g.drow
    # the operators' frame: a ray through (src sin(gam)) off the axis, along (cos th, sin th)
    dist = g.R * torch.sin(gam)
    px, py = (dist * torch.sin(th))[:, None, :], (-dist * torch.cos(th))[:, None, :]
    dx, dy = torch.cos(th)[:, None, :], torch.sin(th)[:, None, :]
    # height of the ray at in-plane distance s from the source: h s / D; s = R cos(gam) - tau
    slope = (h / g.D)[None, :, None]
    pz, dz = slope * (g.R * torch.cos(gam))[None, None, :], -slope
    out = torch.zeros((batch, g.V, rows, g.C), device=DEV)
    for b in range(batch):
        for k in range(e.shape[1]):
            cx, cy, cz, a1, a2, a3, mu = e[b, k].tolist()
            ux, uy, uz = (px - cx) / a1, (py - cy) / a2, (pz - cz) / a3 if rows > 1 else 0.0 * pz
            vx, vy, vz = dx / a1, dy / a2, dz / a3 if rows > 1 else 0.0 * dz
            A = vx * vx + vy * vy + vz * vz
            B = ux * vx + uy * vy + uz * vz
            q = B * B - A * (ux * ux + uy * uy + uz * uz - 1.0)
            out[b] += (mu * 2.0 * torch.sqrt(q.clamp(min=0)) / A * torch.sqrt(1 + slope * slope)).float()
    out += 0.01 * torch.randn(out.shape, generator=gen, device=DEV)
    return out if c.get("rows", 1) > 1 else out[:, :, 0]


def _uneven_shapes(c):
    """Eight protocols between half and the full size, the items cycling through them."""
    got = []
    for k in range(c["batch"] // 3 + (c["batch"] % 3 > 0)):
        s = 0.5 + 0.5 * (k % 8) / 7
        got.append((max(64, round(c["n"] * s)), max(60, round(c["views"] * s)),
                    max(96, round(c["cols"] * s / 4) * 4)))
    return got


UNEVEN_OPS = ("fp", "fbp", "fbp_adjoint")


def _data(c, seed):
    """The case's inputs, from its seed alone."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) * 7919 + 17)
    op, B = c["op"], c["batch"]
    if op == "uneven":
        xs = []
        for k in range(B):
            n, v, co = _uneven_shapes(c)[k // 3]
            g = _Geom(*_param(c, n, v, co))
            make = _sinogram if UNEVEN_OPS[k % 3] == "fbp" else _image
            xs.append(make(g, c, gen, 1)[0].to(torch.bfloat16))
        return {"xs": xs}
    g = _Geom(*_param(c))
    d = {}
    if op in ("fp", "fp_grad", "driver", "fp_cone"):
        d["x"] = _image(g, c, gen, B)
        if op == "fp_grad":
            d["y"] = _sinogram(g, c, gen, B)
    else:
        d["x"] = _sinogram(g, c, gen, B)
        if op.endswith("_grad"):  # the gradient that arrives from a loss on the reconstruction
            body = _image(g, c, gen, B)
            d["gy"] = body + 0.02 * torch.randn(body.shape, generator=gen, device=DEV)
    return d


def prepare(case, seed):
    c, d = case, _data(case, seed)
    st = {"case": c, **d}
    op = c["op"]
    if op == "uneven":
        shapes = _uneven_shapes(c)
        plans = [ct.FanPlan(*_param(c, *s), window=c["window"]) for s in shapes]
        items, st["out"] = [], []
        for k, x in enumerate(d["xs"]):
            plan, kind = plans[k // 3], UNEVEN_OPS[k % 3]
            shape = plan.image_shape if kind == "fbp" else plan.sino_shape
            y = torch.empty(shape, dtype=torch.bfloat16, device=DEV)
            items.append((plan, kind, x, y))
            st["out"].append(y)
        st["batch"] = UnevenBatch(items)
    elif op == "driver":
        st["param"], st["angles"] = _param(c)
        st["x"] = d["x"].cpu().numpy()
    elif "rows" in c:
        st["plan"] = ct.ConePlan(*_param(c), n_rows=c["rows"], nz=c["nz"], window=c["window"],
                                 cosine_weight=c["cosine"])
    else:
        st["plan"] = ct.FanPlan(*_param(c), window=c["window"], short_scan=c["short"],
                                cosine_weight=c["cosine"])
    return st


def run(state):
    c, op = state["case"], state["case"]["op"]
    if op == "uneven":
        state["batch"].run()
        return state["out"]
    if op == "driver":
        B, n = c["batch"], c["n"]
        geom = {"angle": state["angles"], "parameter": state["param"], "vol_shape": [B, n, n],
                "proj_shape": [B, c["views"], c["cols"]]}
        sino = utils.fp_fan_curve(volume=state["x"], **geom)
        return sino, utils.fbp_fan_curve(projection=sino, **geom)
    plan, x = state["plan"], state["x"]
    if op == "fp":
        return plan.fp(x)
    if op == "fbp":
        return plan.fbp(x)
    if op == "fp_cone":
        return plan.fp_cone(x)
    if op == "fdk":
        return plan.fdk(x)
    x = x.detach().requires_grad_()
    if op == "fp_grad":
        sino = ct.forward_project(x, plan)
        (grad,) = torch.autograd.grad(sino, x, sino.detach() - state["y"])
        return sino.detach(), grad
    layer = {"bp_grad": ct.back_project, "fbp_grad": ct.filtered_back_project,
             "fdk_grad": ct.fdk_cone}[op]
    y = layer(x, plan)
    (grad,) = torch.autograd.grad(y, x, state["gy"])
    return y.detach(), grad


def work(case):
    """Bytes: inputs read once, outputs written once.  FLOPs: two per nonzero of the operator's
    matrix (a ray's chord crosses about 2.5 texels' supports per pixel of length; a pixel-view
    takes two detector values, a voxel-view four) and two per tap of the filter."""
    c, op = case, case["op"]
    if op == "uneven":
        each = [dict(c, op=("fp", "fbp", "fbp")[k % 3], batch=1, n=s[0], views=s[1], cols=s[2])
                for k in range(c["batch"]) for s in [_uneven_shapes(c)[k // 3]]]
        w = [work(e) for e in each]
        return {"bytes": sum(x["bytes"] for x in w) / 2, "flops": sum(x["flops"] for x in w)}
    n, V, C, B = c["n"], c["views"], c["cols"], c["batch"]
    rows, nz = c.get("rows", 1), c.get("nz", 1)
    img, sino = n * n * nz * B, V * C * rows * B
    disc = math.pi / 4 * n * n
    # chords of a view's rays, in pixels: the disc's area over the rays' spacing at its centre
    chord = disc / (FAN_MM / C / SDD * SID / (FOV_MM / n))
    ray = 2 * 2.5 * chord * V * rows * B * (2 if rows > 1 else 1)
    back = 2 * disc * V * nz * B * (4 if rows > 1 else 2)
    filt = 2 * sino * C
    by = {"fp": (img + sino, ray), "fp_cone": (img + sino, ray),
          "fp_grad": (2 * img + 2 * sino, 2 * ray), "driver": (2 * img + 2 * sino, ray + back + filt),
          "bp_grad": (2 * img + 2 * sino, 2 * back), "fbp": (img + sino, back + filt),
          "fbp_grad": (2 * img + 2 * sino, 2 * (back + filt)), "fdk": (img + sino, back + filt),
          "fdk_grad": (2 * img + 2 * sino, 2 * (back + filt))}[op]
    return {"bytes": 4 * by[0], "flops": by[1]}


# ---- the operators in float64 ------------------------------------------------------------------


def _march(g, v, rows=0, nz=0):
    """grid_sample coordinates of view v's samples [1, K, C, 2], or [1, K, rows, C, 3] for the
    cone, and the mask and weight of each."""
    ax, ay, sx, sy, n, s0, ds = g.rays(v)
    k = torch.arange(max(1, int(n.max())), device=DEV, dtype=torch.float64)[:, None]
    x, y, live = (ax + k * sx) * (2.0 / g.nx) - 1.0, (ay + k * sy) * (2.0 / g.nx) - 1.0, k < n
    w = 0.125 * g.dx
    if not rows:
        return torch.stack((x, y), -1)[None], (live * w)[None, None]
    h = g.bottom + (torch.arange(rows, device=DEV, dtype=torch.float64) + 0.5) * g.drow
    z = h[None, :, None] * ((s0 + k * ds) / g.D)[:, None, :] * (2.0 / (g.dz * nz))
    x, y = x[:, None, :].expand_as(z), y[:, None, :].expand_as(z)
    w = w * torch.sqrt(1.0 + (h / g.D) ** 2)[None, :, None]
    return torch.stack((x, y, z), -1)[None], (live[:, None, :] * w)[None, None]


def _fp64(g, x, y=None):
    """FP of x [B, n, n]; with y also the transpose applied to FP(x) - y."""
    x = x.double()[None]
    out, grad = [], torch.zeros_like(x)
    for v in range(g.V):
        at, w = _march(g, v)
        xi = x.detach().requires_grad_(y is not None)
        with torch.set_grad_enabled(y is not None):
            p = (F.grid_sample(xi, at, "bilinear", "border", False) * w).sum(2)[0]
        out.append(p.detach())
        if y is not None:
            grad += torch.autograd.grad(p, xi, out[-1] - y[:, v].double())[0]
    return torch.stack(out, 1), grad[0]


def _fp_cone64(g, x, rows):
    x = x.double()[:, None]
    out = torch.empty((x.shape[0], g.V, rows, g.C), device=DEV, dtype=torch.float64)
    for v in range(g.V):
        at, w = _march(g, v, rows, x.shape[2])
        for b in range(x.shape[0]):
            out[b, v] = (F.grid_sample(x[b:b + 1], at, "bilinear", "border", False) * w).sum(2)[0, 0]
    return out


def _bp64(g, s, weighted):
    at, x, y = g.pixels()
    out = torch.zeros((s.shape[0], g.nx * g.nx), device=DEV, dtype=torch.float64)
    acc = torch.zeros((s.shape[0], at.numel()), device=DEV, dtype=torch.float64)
    for v in range(g.V):
        i0, i1, f, w, ok, _ = g.columns(v, x, y)
        acc += ((1 - f) * s[:, v, i0] + f * s[:, v, i1]) * (w if weighted else ok)
    out[:, at] = acc
    return out.reshape(-1, g.nx, g.nx)


def _bpt64(g, img, weighted):
    at, x, y = g.pixels()
    p = img.double().reshape(img.shape[0], -1)[:, at]
    out = torch.zeros((img.shape[0], g.V, g.C), device=DEV, dtype=torch.float64)
    for v in range(g.V):
        i0, i1, f, w, ok, _ = g.columns(v, x, y)
        q = p * (w if weighted else ok)
        out[:, v].index_add_(1, i0, q * (1 - f))
        out[:, v].index_add_(1, i1, q * f)
    return out


def _cone64(g, c, s=None, vol=None):
    """The weighted cone backprojection of s [B, V, rows, C], or its transpose of vol."""
    at, x, y = g.pixels()
    rows, nz = c["rows"], c["nz"]
    z = g.dz * (torch.arange(nz, device=DEV, dtype=torch.float64) + 0.5 - 0.5 * nz)
    B = s.shape[0] if vol is None else vol.shape[0]
    if vol is None:
        acc = torch.zeros((B, nz, at.numel()), device=DEV, dtype=torch.float64)
    else:
        acc = torch.zeros((B, g.V, rows * g.C), device=DEV, dtype=torch.float64)
        p = vol.double().reshape(B, nz, -1)[:, :, at]
    for v in range(g.V):
        i0, i1, f, w, _, U = g.columns(v, x, y)
        r = (z[:, None] * g.D / U - g.bottom) / g.drow - 0.5
        b = torch.floor(r)
        fr = r - b
        r0, r1 = b.long().clamp(0, rows - 1), (b.long() + 1).clamp(0, rows - 1)
        for q, i, m in ((r0, i0, (1 - fr) * (1 - f)), (r0, i1, (1 - fr) * f), (r1, i0, fr * (1 - f)),
                        (r1, i1, fr * f)):
            idx, m = (q * g.C + i).reshape(-1), m * w
            for k in range(B):
                if vol is None:
                    acc[k] += s[k, v].reshape(-1)[idx].reshape(m.shape) * m
                else:
                    acc[k, v].index_add_(0, idx, (p[k] * m).reshape(-1))
    if vol is not None:
        return acc.reshape(B, g.V, rows, g.C)
    out = torch.zeros((B, nz, g.nx * g.nx), device=DEV, dtype=torch.float64)
    out[:, :, at] = acc
    return out.reshape(B, nz, g.nx, g.nx)


def _filtered(g, c, s):
    """Pre-weights and the ramp filter of [B, V, (rows,) C]."""
    w = g.preweights(c)
    s = s.double()
    if w is not None:
        s = s * (w if s.dim() == 4 else w[:, 0])
    return s @ g.toeplitz(c["window"])


def _filtered_t(g, c, s):
    w = g.preweights(c)
    s = s @ g.toeplitz(c["window"])
    return s if w is None else s * (w if s.dim() == 4 else w[:, 0])


def exact(case, seed):
    c, op = case, case["op"]
    with torch.no_grad():
        d = _data(c, seed)
        if op == "uneven":
            out = []
            for k, x in enumerate(d["xs"]):
                g = _Geom(*_param(c, *_uneven_shapes(c)[k // 3]))
                x = x[None]
                out.append((_fp64(g, x)[0] if k % 3 == 0 else
                            _bp64(g, _filtered(g, c, x), True) if k % 3 == 1 else
                            _filtered_t(g, c, _bpt64(g, x, True)))[0])
            return out
        g = _Geom(*_param(c))
        x = d["x"]
        if op == "fp":
            return _fp64(g, x)[0]
        if op == "fp_grad":
            return _fp64(g, x, d["y"])
        if op == "driver":
            s = _fp64(g, x)[0]
            return s, _bp64(g, _filtered(g, c, s), True)
        if op == "fp_cone":
            return _fp_cone64(g, x, c["rows"])
        if op == "bp_grad":
            return _bp64(g, x.double(), False), _bpt64(g, d["gy"], False)
        if op in ("fbp", "fbp_grad"):
            y = _bp64(g, _filtered(g, c, x), True)
            return y if op == "fbp" else (y, _filtered_t(g, c, _bpt64(g, d["gy"], True)))
        y = _cone64(g, c, s=_filtered(g, c, x))
        return y if op == "fdk" else (y, _filtered_t(g, c, _cone64(g, c, vol=d["gy"])))
