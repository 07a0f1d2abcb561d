"""The work that users of this framework have it do, as measurable cases.

Every case goes through the public entry points (Projector2D / Projector3D,
the FBP_CUDA / SIRT_CUDA / SIRT3D_CUDA algorithm objects, projector.fdk, the
autograd projectors).  Inputs are synthetic scans of random balls: the volume
holds the balls, the projections their exact chord lengths plus measurement
noise, so that the projections are dense as a detector's are.

`exact` restates the models in 64 bits with plain torch: the ray-driven forward
projection (bilinear samples of the slices of a ray's dominant axis), the
voxel-driven backprojection (bilinear detector samples with the view's weight),
the ramp filter as a zero-padded FFT product, and SIRT's recurrence.
"""
import importlib
import math

import numpy as np
import torch

astra = importlib.import_module("astra-toolbox_b200")
autograd = importlib.import_module("astra-toolbox_b200.autograd")

F64 = torch.float64
DTYPES = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # The smallest call: one thumbnail slice, both directions, as an
        # iterative program or a notebook issues it.  Launches count.
        {"name": "slice-parallel-128", "op": "project2d", "geom": "parallel", "rows": 128, "cols": 128, "views": 180,
         "dets": 192},
        # An ordinary synchrotron slice: many views, a megapixel.
        {"name": "slice-parallel-1024", "op": "project2d", "geom": "parallel", "rows": 1024, "cols": 1024,
         "views": 1440, "dets": 1536},
        # A fan-beam slice with odd sizes everywhere.
        {"name": "slice-fan-odd", "op": "project2d", "geom": "fanflat", "rows": 513, "cols": 700, "views": 401,
         "dets": 911},
        # Filtered backprojection of one slice through the algorithm object.
        {"name": "fbp-parallel-512", "op": "fbp2d", "geom": "parallel", "rows": 512, "cols": 512, "views": 720,
         "dets": 768},
        # SIRT of a small slice: twenty dependent pairs of short launches.
        {"name": "sirt-parallel-256", "op": "sirt2d", "geom": "parallel", "rows": 256, "cols": 256, "views": 180,
         "dets": 384, "iterations": 20},
        # A small cone-beam volume (a preview, a training sample).
        {"name": "cone-128", "op": "project3d", "geom": "cone", "nx": 128, "ny": 128, "nz": 128, "views": 180,
         "du": 192, "dv": 192, "dtype": "float32"},
        # The headline scan: a full circular cone-beam acquisition.
        {"name": "cone-512", "op": "project3d", "geom": "cone", "nx": 512, "ny": 512, "nz": 512, "views": 720,
         "du": 832, "dv": 832, "dtype": "float32"},
        # FDK of an ordinary scan.
        {"name": "fdk-256", "op": "fdk", "geom": "cone", "nx": 256, "ny": 256, "nz": 256, "views": 360,
         "du": 416, "dv": 416},
        # A calibrated scanner: per-view vectors with jittered, tilted
        # detectors, ragged sizes (the scan type of the large vector workload).
        {"name": "vec-jitter-odd", "op": "project3d", "geom": "cone_vec", "nx": 301, "ny": 320, "nz": 259,
         "views": 333, "du": 403, "dv": 357, "dtype": "float32"},
        # Parallel-beam volume in half storage.
        {"name": "parallel3d-half", "op": "project3d", "geom": "parallel3d", "nx": 256, "ny": 240, "nz": 256,
         "views": 300, "du": 384, "dv": 264, "dtype": "float16"},
        # A training step's data term: forward projection and its exact
        # adjoint through autograd.
        {"name": "adjoint-cone-192", "op": "adjoint", "geom": "cone", "nx": 192, "ny": 192, "nz": 192, "views": 240,
         "du": 288, "dv": 288},
        # Iterative cone-beam reconstruction.
        {"name": "sirt3d-cone-200", "op": "sirt3d", "geom": "cone", "nx": 200, "ny": 200, "nz": 192, "views": 200,
         "du": 300, "dv": 288, "iterations": 5},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["project2d", "project2d", "project2d", "fbp2d", "sirt2d", "project3d", "project3d", "project3d",
                     "project3d", "fdk", "adjoint", "sirt3d"])
    if op in ("project2d", "fbp2d", "sirt2d"):
        n = _log(rng, 64, 256 if op == "sirt2d" else 1024)
        c = {"op": op, "geom": "parallel" if op == "fbp2d" else rng.choice(["parallel", "fanflat"]),
             "rows": max(48, int(n * rng.uniform(0.7, 1.0))), "cols": n, "views": _log(rng, 60, 1440),
             "dets": int(n * rng.uniform(1.2, 1.6))}
        if op == "sirt2d":
            c.update(views=_log(rng, 60, 360), iterations=rng.randint(2, 20))
        return c
    top = {"project3d": 400, "fdk": 400, "adjoint": 256, "sirt3d": 256}[op]
    n = _log(rng, 64, top)
    geom = rng.choice(["cone", "cone", "cone_vec", "parallel3d"]) if op == "project3d" else "cone"
    mag = 1.05 if geom == "parallel3d" else 1.3
    c = {"op": op, "geom": geom, "nx": n, "ny": max(48, int(n * rng.uniform(0.8, 1.0))),
         "nz": max(32, int(n * rng.uniform(0.5, 1.0))), "views": _log(rng, 45, 500), "du": int(n * mag * rng.uniform(1.0, 1.3))}
    c["dv"] = int(c["nz"] * mag * rng.uniform(0.9, 1.2))
    if op == "project3d":
        c["dtype"] = rng.choice(["float32", "float32", "float32", "float16", "bfloat16"])
    if op == "sirt3d":
        c.update(views=_log(rng, 45, 250), iterations=rng.randint(1, 5))
    return c


def _is3d(case):
    return "nz" in case


def work(case):
    """Bytes: each input read and each output written once.  Operations: per
    sample of a forward projection its position and interpolation (2D 5, 3D
    10), per pixel or voxel update of a backprojection its projection,
    interpolation and weight (2D 8, 3D 20)."""
    if _is3d(case):
        vox = case["nx"] * case["ny"] * case["nz"]
        rays = case["views"] * case["du"] * case["dv"]
        fp, bp = rays * min(case["nx"], case["ny"]) * 10, vox * case["views"] * 20
    else:
        vox = case["rows"] * case["cols"]
        rays = case["views"] * case["dets"]
        fp, bp = rays * min(case["rows"], case["cols"]) * 5, vox * case["views"] * 8
    size = 2 if case.get("dtype", "float32") != "float32" else 4
    op = case["op"]
    if op in ("project2d", "project3d"):
        return {"bytes": 2 * size * (vox + rays), "flops": fp + bp}
    if op in ("fbp2d", "fdk"):
        return {"bytes": size * (vox + rays), "flops": bp + rays * 10 * math.log2(2 * (case.get("dets") or case["du"]))}
    if op == "adjoint":  # volume and measured data in; projections and gradient out
        return {"bytes": size * (2 * vox + 2 * rays), "flops": 2 * fp}
    it = case["iterations"]
    return {"bytes": size * (vox + rays), "flops": it * (fp + bp)}


def tolerance(case):
    """About four times the distance from `exact` that was measured over the
    listed sizes and drawn ones."""
    kind = case.get("dtype", "float32")
    if kind != "float32":  # one rounding of the output
        return {"rel": 1e-3 if kind == "float16" else 8e-3}
    return {"rel": {
        "project2d": 1.2e-5,  # sample positions of about a thousand pixels in 32 bits
        "project3d": 5e-6,
        # the ramp's outputs are a hundredth of its inputs: their rounding shows
        "fbp2d": 1.2e-4,
        "fdk": 2e-5,
        # the adjoint is applied to A x - b, a hundredth of A x
        "adjoint": 1e-4,
        # rays that graze the grid's edge have line weights of rounding size
        "sirt2d": 5e-4,
        "sirt3d": 2e-5,
    }[case["op"]]}


# ---------------------------------------------------------------------------
# geometries: the framework's dictionaries, and the same scans' per-view vectors
# ---------------------------------------------------------------------------

def _angles(case):
    turn = math.pi if case["geom"] in ("parallel", "parallel3d") else 2 * math.pi
    return np.linspace(0, turn, case["views"], endpoint=False).astype(np.float32)


def _radii(case):
    """Source-origin and origin-detector distances: magnification 1.5 in 2D,
    1.5 on the 3D orbit (the source two volume widths away)."""
    n = case["nx"] if _is3d(case) else max(case["rows"], case["cols"])
    return 2.0 * n, (1.0 if not _is3d(case) or case["geom"] == "cone" else 0.4) * n


def _spacing(case):
    """Detector pixel size: the panel covers the magnified volume."""
    if not _is3d(case):
        return 1.0 if case["geom"] == "parallel" else 1.5
    return 1.0 if case["geom"] == "parallel3d" else 1.2


def _vectors(case):
    """cone_vec rows: a circular orbit whose detector is shifted by N(0, 0.5
    pixels) along both axes and tilted by N(0, 0.1 degrees) in every view."""
    rng = np.random.default_rng(case["views"] * 1000003 + case["du"] * 1009 + case["dv"])
    so, od = _radii(case)
    px = _spacing(case)
    out = np.zeros((case["views"], 12))
    for i, t in enumerate(np.linspace(0, 2 * np.pi, case["views"], endpoint=False)):
        src = np.array([np.sin(t), -np.cos(t), 0.0]) * so
        u, v = np.array([np.cos(t), np.sin(t), 0.0]), np.array([0.0, 0.0, 1.0])
        n = np.cross(u, v)
        a, b = np.deg2rad(rng.normal(0.0, 0.1, 2))
        su, sv = rng.normal(0.0, 0.5, 2) * px
        out[i, 0:3] = src
        out[i, 3:6] = -src / so * od + su * u + sv * v
        out[i, 6:9] = px * (u * np.cos(a) + n * np.sin(a))
        out[i, 9:12] = px * (v * np.cos(b) + n * np.sin(b))
    return out


def _dictionaries(case):
    px = _spacing(case)
    if _is3d(case):
        vg = astra.create_vol_geom(case["ny"], case["nx"], case["nz"])
        if case["geom"] == "cone_vec":
            return astra.create_proj_geom("cone_vec", case["dv"], case["du"], _vectors(case)), vg
        if case["geom"] == "parallel3d":
            return astra.create_proj_geom("parallel3d", px, px, case["dv"], case["du"], _angles(case)), vg
        return astra.create_proj_geom("cone", px, px, case["dv"], case["du"], _angles(case), *_radii(case)), vg
    vg = astra.create_vol_geom(case["rows"], case["cols"])
    if case["geom"] == "fanflat":
        return astra.create_proj_geom("fanflat", px, case["dets"], _angles(case), *_radii(case)), vg
    return astra.create_proj_geom("parallel", px, case["dets"], _angles(case)), vg


def _views(case):
    """(source or ray direction, detector corner, u step[, v step]) of every
    view, float64 arrays of the numbers that the scan is defined by (2D views
    are stored in 32 bits)."""
    px = float(np.float32(_spacing(case)))
    if case["geom"] == "cone_vec":
        w = _vectors(case)
        u, v = w[:, 6:9], w[:, 9:12]
        return w[:, 0:3], w[:, 3:6] - 0.5 * case["dv"] * v - 0.5 * case["du"] * u, u, v
    a = _angles(case).astype(np.float64)
    c, s, zero, one = np.cos(a), np.sin(a), np.zeros_like(a), np.ones_like(a)
    so, od = _radii(case) if case["geom"] in ("cone", "fanflat") else (None, 0.0)

    def turn(x, y):
        return x * c - y * s, x * s + y * c

    sx, sy = turn(0.0, 1.0) if so is None else turn(0.0, -so)
    ux, uy = turn(px, 0.0)
    n = case["du"] if _is3d(case) else case["dets"]
    dx, dy = turn(-0.5 * n * px, od)
    if _is3d(case):
        z = zero - 0.5 * case["dv"] * px
        return (np.stack([sx, sy, zero], 1), np.stack([dx, dy, z], 1), np.stack([ux, uy, zero], 1),
                np.stack([zero, zero, px * one], 1))

    def f(x, y):
        return np.stack([x, y], 1).astype(np.float32).astype(np.float64)

    return f(sx, sy), f(dx, dy), f(ux, uy)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _balls(shape, seed, count=8):
    """Centres (x, y[, z]), radii and densities of balls inside the volume."""
    rng = np.random.default_rng(int(seed))
    ext = np.array(shape[::-1], dtype=np.float64)
    r = rng.uniform(0.05, 0.25, count) * ext.min()
    return rng.uniform(-0.3, 0.3, (count, ext.size)) * ext, r, rng.uniform(0.2, 1.0, count)


def _shapes(case):
    if _is3d(case):
        return (case["nz"], case["ny"], case["nx"]), (case["dv"], case["views"], case["du"])
    return (case["rows"], case["cols"]), (case["views"], case["dets"])


def _volume(case, seed):
    shape, _ = _shapes(case)
    dev = _device()
    centres, radii, dens = _balls(shape, seed)
    axes = [torch.arange(n, device=dev, dtype=torch.float32) - 0.5 * n + 0.5 for n in shape]
    axes[-2] = axes[-2] if _is3d(case) else -axes[-2]  # image rows run downwards
    out = torch.zeros(shape, device=dev)
    for c, r, d in zip(centres, radii, dens):
        q = 0.0
        for k, ax in enumerate(axes):
            view = [1] * len(shape)
            view[k] = -1
            q = q + ((ax - c[len(shape) - 1 - k]) ** 2).view(view)
        out += float(d) * (q <= r * r)
    return out


def _projections(case, seed):
    """Chord lengths of the balls along every ray, plus 0.5 % noise."""
    vshape, pshape = _shapes(case)
    dev = _device()
    views = [torch.tensor(v, device=dev, dtype=torch.float32) for v in _views(case)]
    if not _is3d(case):
        views = [torch.nn.functional.pad(v, (0, 1)) for v in views]
        views.append(torch.zeros_like(views[0]))
    centres, radii, dens = _balls(vshape, seed)
    centres = np.pad(centres, ((0, 0), (0, 3 - centres.shape[1])))
    nv, na, nu = pshape if _is3d(case) else (1,) + pshape
    out = torch.zeros((nv, na, nu), device=dev)
    iu = torch.arange(nu, device=dev, dtype=torch.float32).view(1, 1, nu) + 0.5
    iv = torch.arange(nv, device=dev, dtype=torch.float32).view(nv, 1, 1) + 0.5
    step = max(1, (1 << 24) // (nv * nu))
    for a0 in range(0, na, step):
        src, det, du, dv = (v[a0:a0 + step] for v in views)
        p = [det[None, :, None, k] + iu * du[None, :, None, k] + iv * dv[None, :, None, k] for k in range(3)]
        if case["geom"] in ("parallel", "parallel3d"):
            d = [src[None, :, None, k] for k in range(3)]
            o = p
        else:
            o = [src[None, :, None, k] for k in range(3)]
            d = [p[k] - o[k] for k in range(3)]
        dd = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
        part = out[:, a0:a0 + step]
        for c, r, w in zip(centres, radii, dens):
            m = [float(c[k]) - o[k] for k in range(3)]
            t = (m[0] * d[0] + m[1] * d[1] + m[2] * d[2]) / dd
            q = sum((m[k] - t * d[k]) ** 2 for k in range(3))
            part += 2.0 * float(w) * torch.sqrt(torch.clamp(float(r * r) - q, min=0.0))
    gen = torch.Generator(device=dev).manual_seed(int(seed) + 17)
    out += 0.005 * float(out.max()) * torch.randn(out.shape, generator=gen, device=dev)
    return out.view(pshape)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

class _Reconstruction:
    """An algorithm object with its data objects, released with the state."""

    def __init__(self, kind, data, pg, vg, proj, vol):
        self.data = data
        self.ids = [data.create("-sino", pg, proj), data.create("-vol", vg, vol)] if data is astra.data2d else \
            [data.create("-proj3d", pg, proj), data.create("-vol", vg, vol)]
        cfg = astra.astra_dict(kind)
        cfg["ProjectionDataId"], cfg["ReconstructionDataId"] = self.ids
        self.id = astra.algorithm.create(cfg)

    def __del__(self):
        astra.algorithm.delete(self.id)
        for i in self.ids:
            self.data.delete(i)


def prepare(case, seed):
    pg, vg = _dictionaries(case)
    op = case["op"]
    vshape, pshape = _shapes(case)
    dev = _device()
    st = {"op": op}
    if op in ("project2d", "project3d"):
        t = DTYPES[case.get("dtype", "float32")]
        st["projector"] = (astra.Projector3D if _is3d(case) else astra.Projector2D)(pg, vg)
        st["vol"], st["proj"] = _volume(case, seed).to(t), _projections(case, seed).to(t)
        st["fp"] = torch.empty(pshape, device=dev, dtype=t)
        st["bp"] = torch.empty(vshape, device=dev, dtype=t)
    elif op == "fdk":
        st["projector"] = astra.Projector3D(pg, vg)
        st["proj"], st["out"] = _projections(case, seed), torch.empty(vshape, device=dev)
    elif op == "adjoint":
        st["projector"] = astra.Projector3D(pg, vg)
        st["vol"], st["data"] = _volume(case, seed).requires_grad_(True), _projections(case, seed)
    else:
        # linked tensors: the data objects work on the user's own memory
        link = astra.data3d if _is3d(case) else astra.data2d
        st["proj"], st["out"] = _projections(case, seed), torch.zeros(vshape, device=dev)
        kind = {"fbp2d": "FBP_CUDA", "sirt2d": "SIRT_CUDA", "sirt3d": "SIRT3D_CUDA"}[op]
        st["rec"] = _Reconstruction(kind, _Linked(link), pg, vg, st["proj"], st["out"])
        st["iterations"] = case.get("iterations", 1)
    return st


class _Linked:
    """data2d / data3d whose objects use the given tensors in place."""

    def __init__(self, module):
        self.module = module

    def create(self, kind, geometry, tensor):
        return self.module.link(kind, geometry, tensor)

    def delete(self, i):
        self.module.delete(i)


def run(st):
    op = st["op"]
    if op in ("project2d", "project3d"):
        st["projector"].fp(st["vol"], st["fp"])
        st["projector"].bp(st["proj"], st["bp"])
        return {"fp": st["fp"], "bp": st["bp"]}
    if op == "fdk":
        return {"volume": astra.projector.fdk(st["projector"], st["proj"], st["out"])}
    if op == "adjoint":
        y = autograd.forward_project(st["vol"], st["projector"])
        grad, = torch.autograd.grad(y, st["vol"], y.detach() - st["data"])
        return {"projections": y.detach(), "gradient": grad}
    if op in ("sirt2d", "sirt3d"):
        st["out"].zero_()  # from zero, as a reconstruction starts
    astra.algorithm.run(st["rec"].id, st["iterations"])
    return {"volume": st["out"]}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _sample(plane, q1, q2):
    """Bilinear samples of plane[q2][q1] at element coordinates, zero outside."""
    h, w = plane.shape
    grid = torch.stack([2 * q1 / (w - 1) - 1, 2 * q2 / (h - 1) - 1], dim=-1)
    return torch.nn.functional.grid_sample(plane[None, None], grid[None], mode="bilinear", padding_mode="zeros",
                                           align_corners=True)[0, 0]


class _Exact3D:
    def __init__(self, case):
        self.dev = _device()
        self.cone = case["geom"] != "parallel3d"
        self.src, self.det, self.u, self.v = (torch.tensor(x, device=self.dev, dtype=F64) for x in _views(case))
        self.nu, self.nv, self.na = case["du"], case["dv"], case["views"]
        self.shape = (case["nz"], case["ny"], case["nx"])
        # the axis along which a view's central ray is longest, in 32 bits
        d = (self.src - (self.det + 0.5 * self.nu * self.u + 0.5 * self.nv * self.v)) if self.cone else self.src
        d = d.to(torch.float32).abs()
        self.axis = torch.where((d[:, 0] >= d[:, 1]) & (d[:, 0] >= d[:, 2]), 0,
                                torch.where((d[:, 1] >= d[:, 0]) & (d[:, 1] >= d[:, 2]), 1, 2)).tolist()

    def _groups(self):
        step = max(1, (1 << 24) // (self.nu * self.nv))
        for ax in (0, 1, 2):
            sel = [i for i, k in enumerate(self.axis) if k == ax]
            for k in range(0, len(sel), step):
                yield ax, sel[k:k + step]

    def _lines(self, ax, sel):
        """Slopes, offsets and length factor of the rays of the views sel."""
        iu = torch.arange(self.nu, device=self.dev, dtype=F64).view(1, 1, -1) + 0.5
        iv = torch.arange(self.nv, device=self.dev, dtype=F64).view(-1, 1, 1) + 0.5
        perm = ((0, 1, 2), (1, 0, 2), (2, 0, 1))[ax]
        p = [self.det[sel, k][None, :, None] + iu * self.u[sel, k][None, :, None] + iv * self.v[sel, k][None, :, None]
             for k in perm]
        s = [self.src[sel, k][None, :, None] for k in perm]
        d = [s[k] - p[k] for k in range(3)] if self.cone else s
        a1, a2 = (d[k] / d[0] + 0 * p[0] for k in (1, 2))
        o = s if self.cone else p
        b1, b2 = o[1] - a1 * o[0], o[2] - a2 * o[0]
        n = self.shape[::-1]
        n0, n1, n2 = (n[k] for k in perm)
        b1, b2 = (b + 0.5 * m - 0.5 for b, m in ((b1, n1), (b2, n2)))
        flat = [t.reshape(-1, self.nu) for t in (a1, a2, b1, b2)]
        return flat, n0, torch.sqrt(1 + a1 * a1 + a2 * a2)

    def fp(self, vol, grad_of=None):
        """A vol; with grad_of, A^T grad_of (vol gives the shape only)."""
        out = torch.zeros((self.nv, self.na, self.nu), device=self.dev, dtype=F64)
        back = torch.zeros(self.shape, device=self.dev, dtype=F64) if grad_of is not None else None
        for ax, sel in self._groups():
            (a1, a2, b1, b2), n0, length = self._lines(ax, sel)
            acc = torch.zeros_like(a1)
            g = (grad_of[:, sel] * length).reshape(-1, self.nu) if grad_of is not None else None
            for s in range(n0):
                x = s - 0.5 * n0 + 0.5
                cut = (slice(None),) * (2 - ax) + (s,)
                if g is None:
                    acc += _sample(vol[cut], a1 * x + b1, a2 * x + b2)
                else:
                    plane = torch.zeros_like(back[cut]).requires_grad_(True)
                    back[cut] += torch.autograd.grad(_sample(plane, a1 * x + b1, a2 * x + b2), plane, g)[0]
            if g is None:
                out[:, sel] = acc.view(self.nv, len(sel), self.nu) * length
        return out if grad_of is None else back

    def bp(self, proj, fdk=False):
        nz, ny, nx = self.shape
        x, y, z = (torch.arange(n, device=self.dev, dtype=F64) - 0.5 * n + 0.5 for n in (nx, ny, nz))
        x, y, z = x.view(1, 1, -1), y.view(1, -1, 1), z.view(-1, 1, 1)
        out = torch.zeros(self.shape, device=self.dev, dtype=F64)

        def dot(f):
            return x * float(f[0]) + y * float(f[1]) + z * float(f[2])

        for a in range(self.na):
            s, d, u, v = (t[a].cpu().numpy() for t in (self.src, self.det, self.u, self.v))
            if self.cone:
                m = s - d
                if fdk:
                    k = 1.0 / np.dot(u, np.cross(v, s))
                else:
                    k = math.sqrt(np.linalg.norm(np.cross(u, v))) / np.dot(u, np.cross(v, m))
                den = 1.0 / ((1.0 if fdk else k * np.dot(u, np.cross(v, s))) - dot(k * np.cross(u, v)))
                pu = (k * np.dot(s, np.cross(v, d)) + dot(k * np.cross(v, m))) * den
                pv = (-k * np.dot(s, np.cross(u, d)) - dot(k * np.cross(u, m))) * den
                w = den * den
            else:
                k = 1.0 / np.dot(s, np.cross(u, v))
                pu = -dot(k * np.cross(s, v)) - k * np.dot(s, np.cross(d, v))
                pv = dot(k * np.cross(s, u)) + k * np.dot(s, np.cross(d, u))
                w = 1.0 / np.linalg.norm(np.cross(u, v))
            q1, q2 = (t.expand(self.shape).reshape(nz * ny, nx) - 0.5 for t in (pu, pv))
            out += _sample(proj[:, a], q1, q2).view(self.shape) * w
        return out


class _Exact2D:
    def __init__(self, case):
        self.dev = _device()
        self.fan = case["geom"] == "fanflat"
        self.views = _views(case)
        self.n = case["dets"]
        self.shape = (case["rows"], case["cols"])

    def fp(self, vol):
        rows, cols = self.shape
        out = torch.zeros((len(self.views[0]), self.n), device=self.dev, dtype=F64)
        i = np.arange(self.n, dtype=np.float64)
        sl = [torch.arange(n, device=self.dev, dtype=F64).view(-1, 1) for n in (cols, rows)]
        for a, (s, d, u) in enumerate(zip(*self.views)):
            p = d[:, None] + (i + 0.5) * u[:, None]
            if self.fan:
                ray = s[:, None] - p
                # which way a ray is marched is decided on its 32-bit extents
                e = [np.abs((i * u[k] + d[k]).astype(np.float32) + np.float32(0.5) - np.float32(s[k])) for k in (0, 1)]
                flat = ~(e[1] > e[0])
            else:
                ray = np.repeat(s[:, None], self.n, 1)
                flat = np.full(self.n, abs(np.float32(s[0])) > abs(np.float32(s[1])))
            for pick, (k, j) in ((flat, (0, 1)), (~flat, (1, 0))):
                if not pick.any():
                    continue
                slope = ray[j, pick] / ray[k, pick]
                off = p[j, pick] - slope * p[k, pick]
                t, b = (torch.tensor(q, device=self.dev, dtype=F64).view(1, -1) for q in (slope, off))
                if k == 0:  # columns are the slices; y points up
                    q2 = 0.5 * rows - (t * (sl[0] - 0.5 * cols + 0.5) + b) - 0.5
                    val = _sample(vol, sl[0].expand(q2.shape), q2)
                else:
                    q1 = (t * (0.5 * rows - sl[1] - 0.5) + b) + 0.5 * cols - 0.5
                    val = _sample(vol, q1, sl[1].expand(q1.shape))
                ln = torch.tensor(np.sqrt(1 + slope ** 2), device=self.dev, dtype=F64)
                out[a, torch.tensor(np.nonzero(pick)[0], device=self.dev)] = val.sum(0) * ln
        return out

    def bp(self, sino):
        rows, cols = self.shape
        x = (torch.arange(cols, device=self.dev, dtype=F64) - 0.5 * cols + 0.5).view(1, -1)
        y = -(torch.arange(rows, device=self.dev, dtype=F64) - 0.5 * rows + 0.5).view(-1, 1)
        out = torch.zeros(self.shape, device=self.dev, dtype=F64)
        pad = torch.nn.functional.pad(sino, (2, 2))
        for a, (s, d, u) in enumerate(zip(*self.views)):
            if self.fan:
                m = s - d
                k = math.hypot(*u) / (u[0] * m[1] - u[1] * m[0])
                w = 1.0 / (k * (u[0] * s[1] - u[1] * s[0]) + x * (k * u[1]) - y * (k * u[0]))
                t = (k * (s[0] * d[1] - s[1] * d[0]) + x * (k * m[1]) - y * (k * m[0])) * w
            else:
                k = u[0] * s[1] - u[1] * s[0]
                t = (x * s[1] - y * s[0] + (d[1] * s[0] - d[0] * s[1])) / k
                w = math.hypot(*s) / abs(k)
            q = torch.clamp(t - 0.5 + 2.0, 0.0, self.n + 2.0)
            lo = torch.floor(q)
            j = lo.long()
            row = pad[a]
            out += (row[j] + (q - lo) * (row[j + 1] - row[j])) * w
        return out


def _ramp(rows):
    """Rows filtered with the ramp's spatial taps (1/2, -2/(pi k)^2 at odd k)."""
    n = rows.shape[-1]
    size = 1 << (2 * n - 1).bit_length()
    k = torch.arange(size, device=rows.device, dtype=F64)
    k = torch.minimum(k, size - k)
    h = torch.where(k % 2 == 1, -2.0 / (math.pi * torch.clamp(k, min=1.0)) ** 2, torch.zeros_like(k))
    h[0] = 0.5
    return torch.fft.irfft(torch.fft.rfft(rows, size) * torch.fft.rfft(h), size)[..., :n]


def _inverse(x):
    return torch.where(x > 1e-6, 1.0 / torch.clamp(x, min=1e-6), torch.zeros_like(x))


def exact(case, seed):
    if _is3d(case):
        samples = case["nx"] * case["du"] * case["dv"] * case["views"] * case.get("iterations", 1)
        if samples > 4e10:
            return None
    op = case["op"]
    model = _Exact3D(case) if _is3d(case) else _Exact2D(case)
    t = DTYPES[case.get("dtype", "float32")]
    proj = _projections(case, seed).to(t).to(F64)
    if op in ("project2d", "project3d"):
        return {"fp": model.fp(_volume(case, seed).to(t).to(F64)), "bp": model.bp(proj)}
    if op == "adjoint":
        y = model.fp(_volume(case, seed).to(F64))
        return {"projections": y, "gradient": model.fp(None, grad_of=y - proj)}
    if op == "fbp2d":
        return {"volume": model.bp(_ramp(proj)) * (math.pi / 2 / case["views"])}
    if op == "fdk":
        px = _spacing(case)
        so, od = _radii(case)
        length = so + od
        u, v = ((torch.arange(n, device=proj.device, dtype=F64) - 0.5 * n + 0.5) * px for n in (case["du"], case["dv"]))
        ray = torch.sqrt(length ** 2 + u.view(1, 1, -1) ** 2 + v.view(-1, 1, 1) ** 2)
        scale = length * length / (px * so) * (math.pi / 2) / case["views"]
        return {"volume": model.bp(_ramp(proj * (scale / ray)), fdk=True)}
    vshape, pshape = _shapes(case)
    line = _inverse(model.fp(torch.ones(vshape, device=proj.device, dtype=F64)))
    pix = _inverse(model.bp(torch.ones(pshape, device=proj.device, dtype=F64)))
    x = torch.zeros(vshape, device=proj.device, dtype=F64)
    for _ in range(case["iterations"]):
        x += pix * model.bp((proj - model.fp(x)) * line)
    return {"volume": x}
