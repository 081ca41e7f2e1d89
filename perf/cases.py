"""Timed workloads of the AFAR solver: what its users have it do, from single small solves to the
largest ones, through the package's public entry points.

A case names a mesh family and its size, a precision policy, a way of driving the solver and the RK3
steps of one pass:

* ``run``    the fields as they were at the start of the pass (device snapshot), ``steps`` steps of
             ``CudaSolver.run`` with the device Courant step, the fields read back: a program that
             writes its fields every ``steps`` steps;
* ``evolve`` the same, stepped as the reference application does it: the Courant step to the host and
             one evolve call for each step;
* ``batch``  several solves of different sizes advanced together by one ``Batch``;
* ``serve``  several requests handed to a resident ``Server`` and waited for.

The initial fields come from the seed alone; meshes and operators belong to the case.  The fields of
the mixed policy are FP32 in the solver, so they are handed on as FP32; its switch flags, decided by
FP32 comparisons of nearly equal numbers all over a smooth flow, are not part of the result.  The
other policies return their flags too.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from afar_cudaeuler2dmixo3rk3solver_gb300 import Batch, CaseConfig, CudaSolver, HostFields, Server, lib, mesh, precompute
from afar_cudaeuler2dmixo3rk3solver_gb300._ffi import FieldPointer, check

FACE_NEIGHBOUR = ("ramp", "ramps", "quads")  # families whose programs use face-neighbour stencils


def listed():
    return [
        # the smallest solve: a coarse vortex, where the launches of a step are all there is
        _case("vortex_1k_mixed", "vortex", 32, "mixed", "run", 20),
        # a small mesh of odd size with triangles and quads, all in FP64
        _case("riemann_2k_fp64", "riemann", 37, "fp64", "run", 20),
        # one compression ramp through the reference-shaped loop: a host round trip for each step
        _case("ramp_11k_evolve_mixed", "ramp", 75, "mixed", "evolve", 20),
        # the accuracy study's vortex on 256 x 256 quads
        _case("vortex_65k_mixed", "vortex", 256, "mixed", "run", 50),
        # the same vortex in a periodic box with the multi-point face flux
        _case("periodic_23k_gauss_fp64", "periodic", 151, "fp64", "run", 5, gauss=True),
        # the reference's own case (corner flow, its settings) in its own arithmetic and loop
        _case("corner_250k_evolve_ref", "corner", 500, "ref", "evolve", 5),
        # Mach 3 forward step, half a million triangles: all FP64
        _case("step_500k_fp64", "step", 250_000, "fp64", "run", 5),
        # the same through the reference-shaped loop in the fast policy
        _case("step_500k_evolve_mixed", "step", 250_000, "mixed", "evolve", 20),
        # the headline workload: Mach 3 forward step, two million triangles
        _case("step_2m_mixed", "step", 1_000_000, "mixed", "run", 20),
        # the largest: four-quadrant Riemann problem on four million quads and triangles
        _case("riemann_4m_mixed", "riemann", 1766, "mixed", "run", 10),
        # a parameter study: compression ramps of many sizes stepped together
        _case("ramps_24_batch_mixed", "ramps", 24, "mixed", "batch", 20),
        # requests to a resident server: set-up, stepping and read-back of small solves
        _case("quads_6_serve_mixed", "quads", 6, "mixed", "serve", 50),
    ]


def _case(name, family, size, policy, drive, steps, gauss=False):
    return {"name": name, "family": family, "size": size, "policy": policy, "drive": drive, "steps": steps,
            "gauss": gauss}


#: The sizes that each family is used at (quads a side, points, solves).
RANGES = {"vortex": (24, 640), "riemann": (20, 1200), "ramp": (20, 320), "periodic": (16, 160), "corner": (40, 500),
          "step": (1_500, 250_000), "ramps": (2, 24), "quads": (1, 6)}


def draw(rng):
    family = rng.choice(list(RANGES))
    lo, hi = RANGES[family]
    size = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if family == "ramps":
        policy, drive = rng.choice(("mixed", "mixed", "fp64")), "batch"
    elif family == "quads":
        policy, drive = "mixed", "serve"
    else:
        # a periodic mesh has no ref form
        policy = rng.choice(("mixed", "mixed", "fp64") + (() if family == "periodic" else ("ref",)))
        drive = rng.choice(("run", "evolve"))
    gauss = family in ("periodic", "vortex") and size <= 160 and policy != "ref" and rng.random() < 0.4
    c = _case("", family, size, policy, drive, rng.randint(4, 12), gauss)
    del c["name"]
    return c


# ------------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _bundle(family, size, part, policy, gauss):
    """Mesh, settings and host operators of one solve (the FP64 weights too where they are used)."""
    order = "edgeNeighbour"
    cfl, R, extra = 0.3, mesh.R_GAS, {}
    if family == "vortex":
        m = mesh.vortex_box(size)
    elif family == "periodic":
        m = mesh.periodic_quad_grid(size, size, 0.0, 10.0, 0.0, 10.0)
    elif family == "riemann":
        m = mesh.riemann_mixed(size, seed=1)
    elif family == "step":
        m, cfl = mesh.forward_step_triangles(size, seed=0), 0.2
    elif family == "corner":
        # the reference case's settings; its Courant step leaves the inlet out, so a smaller number
        m, cfl, extra = mesh.corner_flow(size), 0.1, dict(Cv=1.7857142857, cOrder=7, fOrder=5)
        R = 0.7142857
    elif family == "ramp":
        m = mesh.wedge_quads(2 * size, size, 12.5)
    elif family == "ramps":  # 5 to 200 thousand cells, 5 to 20 degrees
        r = np.random.default_rng(100 + part)
        ny = max(8, int(round(math.sqrt(math.exp(r.uniform(math.log(5e3), math.log(2e5))) / 2.0))))
        m = mesh.wedge_quads(2 * ny, ny, float(r.uniform(5.0, 20.0)))
    else:  # quads: requests of 10 to 50 thousand cells
        n = 100 + 37 * (part % 4)
        m = mesh.quad_grid(n, n, 0.0, 1.2, 0.0, 1.0)
    if family in FACE_NEIGHBOUR:
        order = "faceNeighbour"
    cfg = CaseConfig(R=R, CFL=cfl, stencilType=order, **extra)
    W, Wb = mesh.uniform_fields(m, 1.0, 0.0, 0.0, 1.0)
    return m, cfg, precompute(m, cfg, W, Wb, want_rbf64=True, device=None if gauss else 0, gauss_flux=gauss)


def _wave(xy, rng, amplitude):
    """A smooth disturbance: four plane waves of random direction and phase."""
    out = np.zeros(xy.shape[0])
    for k in range(4):
        a, ph = rng.uniform(0.0, 2.0 * math.pi, 2)
        out += np.sin((k + 2.0) * (math.cos(a) * xy[:, 0] + math.sin(a) * xy[:, 1]) + ph)
    return 1.0 + 0.25 * amplitude * out


def _fields(family, m, cfg, seed, part):
    """Primitive fields (p, Ux, Uy, T) of the cells and the boundary ghosts."""
    rng = np.random.default_rng([seed, part])
    xy, xb = m.cell_centres(), m.boundary_face_centres()
    if family in ("vortex", "periodic"):
        c = rng.uniform(-0.5, 0.5, 2) + (0.0 if family == "vortex" else 5.0)
        kw = dict(strength=float(rng.uniform(4.0, 5.5)), xc=float(c[0]), yc=float(c[1]))
        return mesh.vortex_fields(xy, **kw), mesh.vortex_fields(xb, **kw)
    if family in ("ramp", "ramps"):
        u0 = float(rng.uniform(1.5, 4.0)) * math.sqrt(1.4)
        at = dict(xc=0.5, yc=0.6, u0=u0, v0=0.0)
        return (mesh.vortex_fields(xy, strength=float(rng.uniform(1.0, 5.0)), **at),
                mesh.vortex_fields(xb, strength=0.0, **at))
    if family in ("riemann", "quads"):
        W, _ = mesh.riemann_fields(m)
        W *= _wave(xy, rng, 0.02)[:, None]
        return W, W[m.owner[m.n_internal_faces:]]
    state = (1.0, 3.0, 0.0, 1.0) if family == "step" else (1.0, 0.0, 0.0, 1.0)
    W, Wb = mesh.uniform_fields(m, *state)
    W[:, 0] *= _wave(3.0 * xy, rng, 0.04)
    W[:, 3] *= _wave(3.0 * xy, rng, 0.04)
    W[:, 1] += 0.05 * (_wave(3.0 * xy, rng, 1.0) - 1.0)
    W[:, 2] += 0.05 * (_wave(3.0 * xy, rng, 1.0) - 1.0)
    if family == "corner":
        inlet = [p for p in m.patches if p[0] == "inlet"][0]
        at = inlet[2] - m.n_internal_faces
        Wb[at:at + inlet[3]] = (30.05945, 4.07795, 0.0, 5.97677)
    return W, Wb


def _parts(case):
    """The solves of a case: (settings, host fields ready to upload) of each."""
    out = []
    for part in range(case["size"] if case["family"] in ("ramps", "quads") else 1):
        m, cfg, hf = _bundle(case["family"], 0 if case["family"] in ("ramps", "quads") else case["size"], part,
                             case["policy"], case["gauss"])
        W, Wb = _fields(case["family"], m, cfg, case["seed"], part)
        U = mesh.conserved_from_primitive(W, cfg.R, cfg.Cv)
        out.append((m, cfg, HostFields(hf.sizes, dict(hf.a, FD=np.concatenate([W, Wb]), cFD=U, cFDold=U), hf.period)))
    return out


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = dict(case, seed=seed)
    s.parts = _parts(s.case)
    s.solvers, s.out, s.batch = [], [], None
    if case["drive"] == "serve":
        s.server = Server(case["policy"], chunk_steps=25)
        return s
    for _, cfg, hf in s.parts:
        v = CudaSolver(hf, cfg, policy=case["policy"], gauss_flux=case["gauss"])
        if case["drive"] == "batch":
            v.set_step_params()
        v.save()
        n = hf.nc + hf.nb
        s.solvers.append(v)
        s.out.append((torch.empty((n, 4), dtype=torch.float64, pin_memory=True),
                      torch.empty(2 * n, dtype=torch.int8, pin_memory=True)))
    if case["drive"] == "batch":
        s.batch = Batch(case["policy"])
        for v in s.solvers:
            s.batch.add(v)
    return s


def _read(v, out):
    """The fields and flags into the program's own pinned arrays (copyFieldDataDeviceToHost)."""
    fp = FieldPointer()
    fp.FD = ctypes.c_void_p(out[0].data_ptr())
    fp.shockIndicator = ctypes.c_void_p(out[1].data_ptr())
    check(lib().afar_copyFieldDataDeviceToHost(ctypes.byref(fp), v.h, v.fields.nc, v.fields.nb))


def _result(policy, FD, flags):
    if policy == "mixed":
        return {"FD": (FD if torch.is_tensor(FD) else torch.from_numpy(FD)).to(torch.float32)}
    return {"FD": FD, "flags": flags}


def run(s):
    case, got = s.case, []
    if case["drive"] == "serve":
        ids = [s.server.submit(hf, cfg, n_steps=case["steps"]) for _, cfg, hf in s.parts]
        for i in ids:
            FD, flags, _ = s.server.wait(i)
            got.append(_result(case["policy"], FD, flags))
        return got
    for v in s.solvers:
        v.restore()
    if s.batch is not None:
        s.batch.run(case["steps"])
    else:
        v = s.solvers[0]
        if case["drive"] == "run":
            v.run(case["steps"])
        else:
            for _ in range(case["steps"]):
                v.evolve(v.set_delta_t())
    for v, out in zip(s.solvers, s.out):
        _read(v, out)
        got.append(_result(case["policy"], *out))
    return got


# ------------------------------------------------------------------------------------ work
def work(case):
    """Compulsory bytes and operations of the stepping: per stage the state, its operators and the
    geometry read once and the new state written once (no intermediates), plus the Courant step; the
    operations of reconstruction, flux and update counted from their formulas."""
    n = case["size"]
    tri = 0.0
    if case["family"] in ("vortex", "periodic", "corner"):
        cells = float(n * n)
    elif case["family"] == "ramp":
        cells = 2.0 * n * n
    elif case["family"] == "step":
        cells, tri = 2.0 * n, 1.0
    elif case["family"] == "riemann":
        split = math.pi * 0.3 ** 2
        cells = n * n * (1.0 + split)
        tri = 2.0 * split / (1.0 + split)
    elif case["family"] == "ramps":
        cells = 0.0
        for part in range(n):
            r = np.random.default_rng(100 + part)
            ny = max(8, int(round(math.sqrt(math.exp(r.uniform(math.log(5e3), math.log(2e5))) / 2.0))))
            cells += 2.0 * ny * ny
    else:
        cells = float(sum((100 + 37 * (p % 4)) ** 2 for p in range(n)))
    faces_per_cell = 4.0 - tri
    faces = 0.5 * faces_per_cell * cells
    S = faces_per_cell if case["family"] in FACE_NEIGHBOUR else 8.0 + 5.0 * tri
    w = 4.0 if case["policy"] == "mixed" else 8.0  # primitive words
    o = 8.0 if case["policy"] == "fp64" else 4.0  # operator words
    points = 2.0 if case["gauss"] else 0.0
    stage = cells * (8 * w + 120 + 2 * faces_per_cell * o + 4 * S + 4 * faces_per_cell + 2)
    stage += faces * (48 + 2 * (S + 1) * o * (1.0 + points))
    step = 3 * stage + cells * (4 * w + 16) + 48 * faces
    flops = 3 * (cells * (S * (4 + 8 * faces_per_cell * (1.0 + points)) + 30 * faces_per_cell + 60)
                 + faces * 330 * max(1.0, points))
    return {"bytes": case["steps"] * step + cells * 4 * w, "flops": case["steps"] * flops}


# ------------------------------------------------------------------------------------ 64-bit values
def exact(case, seed):
    """The same steps in plain 64-bit torch, from the same mesh, weights and initial fields."""
    case = dict(case, seed=seed)
    res = []
    for m, cfg, hf in _parts(case):
        FD = _Scheme(hf, cfg, case["policy"], case["gauss"]).run(case["steps"])
        res.append({"FD": FD, "flags": None} if case["policy"] != "mixed" else {"FD": FD})
    return res


class _Scheme:
    """The AFAR scheme (least-squares gradients, O3 face values, troubled-cell and BVD switches, Roe or
    KFVS face flux, three-stage Runge-Kutta with the reference's truncated coefficients)."""

    def __init__(self, hf, cfg, policy, gauss):
        a, z, dev = hf.a, hf.sizes, torch.device("cuda" if torch.cuda.is_available() else "cpu")
        f8 = lambda x: torch.as_tensor(np.ascontiguousarray(x, dtype=np.float64), device=dev)  # noqa: E731
        i8 = lambda x: torch.as_tensor(np.ascontiguousarray(x, dtype=np.int64), device=dev)  # noqa: E731
        self.nc, self.nf, self.nb = hf.nc, hf.nf, hf.nb
        nc, nf, S, M = hf.nc, hf.nf, z["maxStencilSize"], z["maxCompactStencilSize"]
        self.R, self.Cv, self.cfl = cfg.R, cfg.Cv, cfg.CFL
        self.pi = math.pi if policy == "fp64" else 3.141593
        self.px, self.py = hf.period
        self.S, self.M = S, M
        nS, nM = i8(a["stencilSize"]), i8(a["compactStencilSize"])
        local, halo, block = i8(a["localStencil"]).view(nc, S), i8(a["extendStencil"]), 128
        at = torch.arange(nc, device=dev) // block
        width = z["maxLocalBlockStencilSize"] - block
        inside = at[:, None] * block + local
        outside = halo[(at[:, None] * width + (local - block).clamp(min=0)).clamp(max=max(0, halo.numel() - 1))] \
            if halo.numel() else inside
        self.st = torch.where(local < block, inside, outside)
        self.in_s = torch.arange(S, device=dev)[None, :] < nS[:, None]
        self.in_m = torch.arange(M, device=dev)[None, :] < nM[:, None]
        own = torch.arange(nc, device=dev)[:, None]
        self.st = torch.where(self.in_s, self.st, own)
        cf = i8(a["cellFaces"]).view(nc, M)
        self.sign = torch.where(self.in_m, torch.sign(cf), 0).double()
        self.face = torch.where(self.in_m, cf.abs() - 1, 0)
        self.inner = self.in_m & (self.face < nf)
        self.side = (cf < 0).long()
        face, cell = f8(a["FACE"]), f8(a["CELL"])
        self.fx, self.fy, self.mag, self.sx, self.sy = (face[:, k].contiguous() for k in range(5))
        self.V = f8(a["cellVolume"])
        nb2 = i8(a["neighbour"]).view(nf, 2)
        self.own, self.nei = nb2[:, 0], nb2[:, 1]
        self.bown, self.btype = i8(a["boundaryFaceNeiLabel"]), i8(a["boundaryFacesType"])
        cx, cy = cell[:, 0].contiguous(), cell[:, 1].contiguous()
        self.cx, self.cy = cx, cy
        # least-squares rows
        dx = [self.wrap(cx[self.st[:, i]] - cx[:nc], self.px) * self.in_m[:, i] for i in range(M)]
        dy = [self.wrap(cy[self.st[:, i]] - cy[:nc], self.py) * self.in_m[:, i] for i in range(M)]
        xx, xy, yy = (sum(u * v for u, v in zip(p, q)) for p, q in ((dx, dx), (dx, dy), (dy, dy)))
        det = xx * yy - xy * xy
        self.m1 = [(yy * u - xy * v) / det for u, v in zip(dx, dy)]
        self.m2 = [(-xy * u + xx * v) / det for u, v in zip(dx, dy)]
        self.ofx = [self.wrap(self.fx[self.face[:, i]] - cx[:nc], self.px) for i in range(M)]
        self.ofy = [self.wrap(self.fy[self.face[:, i]] - cy[:nc], self.py) for i in range(M)]
        self.dr = [torch.where(self.inner[:, i], torch.hypot(dx[i], dy[i]), 1.0) for i in range(M)]
        self.fr = [torch.where(self.inner[:, i], torch.hypot(self.ofx[i], self.ofy[i]) / self.dr[i], 0.0)
                   for i in range(M)]
        w = f8(a["RBFbasis64"]).view(nf, 2, 1, S + 1)
        self.points = [(0.0, 0.0, 1.0)]  # offset of each flux point from the face centre, and its weight
        if gauss:
            p, q = f8(a["faceGaussPoints"]), f8(a["faceGaussWeights"])[0]
            self.points = [(self.wrap(p[:, k, 0] - self.fx[:nf], self.px), self.wrap(p[:, k, 1] - self.fy[:nf], self.py),
                            float(q[k] / q.sum())) for k in range(p.shape[1])]
            w = torch.cat([w, f8(a["RBFbasisGauss64"]).view(nf, 2, len(self.points), S + 1)], dim=2)
        self.w = w
        self.gauss = gauss
        self.dxo = [self.wrap(self.fx[:nf] - cx[c], self.px) for c in (self.own, self.nei)]
        self.dyo = [self.wrap(self.fy[:nf] - cy[c], self.py) for c in (self.own, self.nei)]
        self.FD, self.U = f8(a["FD"]), f8(a["cFD"])

    @staticmethod
    def wrap(d, period):
        return d - period * torch.round(d / period) if period > 0 else d

    def run(self, steps):
        for _ in range(steps):
            dt, U0 = self.courant(), self.U
            for b1, b2, b3 in ((1.0, 0.0, 1.0), (0.75, 0.25, 0.25), (0.333333, 0.666667, 0.666667)):
                res = self.residual()
                self.U = b1 * U0 + b2 * self.U - b3 * dt * res / self.V[:, None]
                rho, mx, my, E = (self.U[:, k] for k in range(4))
                p = self.R / self.Cv * (E - 0.5 * (mx * mx + my * my) / rho)
                self.FD[: self.nc] = torch.stack([p, mx / rho, my / rho, p / (self.R * rho)], 1)
                self.ghosts()
        return self.FD

    def courant(self):
        o, n, f = self.FD[self.own], self.FD[self.nei], slice(0, self.nf)
        dr = torch.hypot(self.wrap(self.cx[self.nei] - self.cx[self.own], self.px),
                         self.wrap(self.cy[self.nei] - self.cy[self.own], self.py))
        w = torch.hypot(self.dxo[0], self.dyo[0]) / dr
        un = [(v[:, 1] * self.sx[f] + v[:, 2] * self.sy[f]).abs() for v in (o, n)]
        c = torch.sqrt((self.R / self.Cv + 1.0) * self.R * ((1 - w) * o[:, 3] + w * n[:, 3]))
        return (self.cfl * dr * self.mag[f] / ((1 - w) * un[0] + w * un[1] + c * self.mag[f])).min()

    def ghosts(self):
        if not self.nb:
            return
        w, t = self.FD[self.bown], self.btype[:, None]
        nx, ny = self.sx[self.nf:] / self.mag[self.nf:], self.sy[self.nf:] / self.mag[self.nf:]
        un = w[:, 1] * nx + w[:, 2] * ny
        slip = torch.stack([w[:, 0], w[:, 1] - un * nx, w[:, 2] - un * ny, w[:, 3]], 1)
        g = torch.where(t == 4, w, torch.where(t == 2, slip, self.FD[self.nc:]))  # label 6 keeps its state
        for label, v in ((3, (1.0, 3.0, 0.0, 1.0)), (5, (30.05945, 4.07795, 0.0, 5.97677))):
            g = torch.where(t == label, torch.tensor(v, dtype=g.dtype, device=g.device), g)
        self.FD[self.nc:] = g

    def residual(self):
        nc, nf, M = self.nc, self.nf, self.M
        FD, W = self.FD, self.FD[: self.nc]
        gx, gy, hi, lo = torch.zeros_like(W), torch.zeros_like(W), W.clone(), W.clone()
        across = []
        for i in range(M):
            v = FD[self.st[:, i]]
            gx += self.m1[i][:, None] * (v - W)
            gy += self.m2[i][:, None] * (v - W)
            hi = torch.where(self.in_m[:, i:i + 1], torch.maximum(hi, v), hi)
            lo = torch.where(self.in_m[:, i:i + 1], torch.minimum(lo, v), lo)
            across.append(v[:, 0])
        flat = (hi[:, 3] - lo[:, 3]).abs() < 1e-10
        o3 = ((hi - lo).abs() >= 1e-5) & ~flat[:, None]
        lim = torch.full_like(W, 2.0)
        smooth, sound = torch.zeros_like(W[:, 0]), torch.ones_like(flat)
        npts = self.w.shape[2]
        fv = torch.zeros((npts, 2, nf, 4), dtype=W.dtype, device=W.device)
        for i in range(M):
            inn, f, sd = self.inner[:, i], self.face[:, i].clamp(max=max(0, nf - 1)), self.side[:, i]
            for k in range(npts):
                dx, dy = self.ofx[i], self.ofy[i]
                if k:
                    dx, dy = dx + self.points[k - 1][0][f], dy + self.points[k - 1][1][f]
                lin = W + gx * dx[:, None] + gy * dy[:, None]
                w = self.w[f, sd, k]
                val = w[:, :1] * W
                for j in range(self.S):
                    val = val + (w[:, j + 1] * self.in_s[:, j])[:, None] * FD[self.st[:, j]]
                fv[k].view(2 * nf, 4)[(sd * nf + f)[inn]] = torch.where(o3, val, lin)[inn]
                if k == 0:
                    d2 = lin - W
                    d1 = torch.where(lin < W, lo - W, hi - W)
                    y = (0.5 * d1 / (d2 + torch.where(d2 >= 0, 1e-10, -1e-10))).clamp(max=2.0)
                    y = torch.where(d2.abs() >= 1e-5, y, 1.0)
                    lim = torch.where(inn[:, None], torch.minimum(lim, y), lim)
                    jump = ((1 - self.fr[i]) * W[:, 0] + self.fr[i] * across[i] - lin[:, 0]).abs() / self.dr[i]
                    jump = jump + (val[:, 0] <= 0) * 1e20 + (lin[:, 0] <= 0) * 1e20
                    smooth = torch.where(inn, torch.maximum(smooth, jump), smooth)
                    sound = torch.where(inn, lin[:, 3] > 0, sound)
        lim = torch.where(flat[:, None], 1.0, lim.clamp(min=0.0) * sound[:, None])
        bad = (smooth / (0.5 * (hi[:, 0] + lo[:, 0]) * sound + 1e-10) > 1.0) & ~flat
        # the switch: troubled cells of the stencil, the variation across the faces
        flag = torch.zeros(nc + self.nb, dtype=torch.int64, device=W.device)
        flag[:nc] = bad
        near, wide = flag[:nc].clone(), flag[:nc].clone()
        for j in range(self.S):
            got = flag[self.st[:, j]] * self.in_s[:, j]
            wide += got
            if j < M:
                near += got * self.in_m[:, j]
        bj = (2 * lim).clamp(max=1.0)
        tvd, walls = torch.zeros_like(flat), torch.zeros_like(near)
        for i in range(M):
            inn, f, sd = self.inner[:, i], self.face[:, i].clamp(max=max(0, nf - 1)), self.side[:, i]
            walls += self.in_m[:, i] & ~inn
            cur, other = fv[0, sd, f, 3], fv[0, 1 - sd, f, 3]
            t = W[:, 3] + bj[:, 3] * (gx[:, 3] * self.ofx[i] + gy[:, 3] * self.ofy[i])
            less = (t - other).abs() < 0.5 * (cur - other).abs()
            moved = (cur - other).abs() > 1e-10
            tvd = tvd | (inn & less & moved & ((bj[:, 3] < 0.9) | (wide > 0)))
        tvd = tvd | (walls >= 2)
        shock = (near > 0) & (wide > 1)
        vk = ((lim * lim + lim + 1e-10) / (lim * lim + 0.5 + 0.5 * lim + 1e-10)).clamp(max=1.0)
        lim = torch.where(shock[:, None], vk, bj)
        kind = tvd.long() - 2 * shock.long()
        # face flux
        F = torch.zeros((nf + self.nb, 4), dtype=W.dtype, device=W.device)
        kfvs = (kind[self.own] < 0) | (kind[self.nei] < 0)
        for k, (ox, oy, wk) in enumerate(self.points):
            st, td = [], []
            for s, c in enumerate((self.own, self.nei)):
                t = W[c] + lim[c] * (gx[c] * (self.dxo[s] + ox)[:, None] + gy[c] * (self.dyo[s] + oy)[:, None])
                td.append(t)
                st.append(torch.where((kind[c] != 0)[:, None], t, fv[k + 1 if self.gauss else 0, s]))
            F[:nf] += wk * self.flux(st, td, kfvs)
        g = FD[nc:]
        rho = g[:, 0] / (self.R * g[:, 3])
        m = rho * (g[:, 1] * self.sx[nf:] + g[:, 2] * self.sy[nf:])
        h = self.Cv * g[:, 3] + 0.5 * (g[:, 1] ** 2 + g[:, 2] ** 2) + g[:, 0] / rho
        F[nf:] = torch.stack([m, m * g[:, 1] + g[:, 0] * self.sx[nf:], m * g[:, 2] + g[:, 0] * self.sy[nf:], m * h], 1)
        res = torch.zeros_like(W)
        for i in range(M):
            res += self.sign[:, i:i + 1] * F[self.face[:, i]]
        return res

    def flux(self, st, td, kfvs):
        R, Cv, n = self.R, self.Cv, slice(0, self.nf)
        sx, sy, mag = self.sx[n], self.sy[n], self.mag[n]
        nx, ny = sx / mag, sy / mag
        p, ux, uy, T = ([v[:, k] for v in st] for k in range(4))
        rho = [p[s] / (R * T[s]) for s in (0, 1)]
        rt = [t[:, 0] / (R * t[:, 3]) for t in td]
        ke = [0.5 * (ux[s] ** 2 + uy[s] ** 2) for s in (0, 1)]
        h = [Cv * T[s] + ke[s] + p[s] / rho[s] for s in (0, 1)]
        m = sum(0.5 * rho[s] * (ux[s] * sx + uy[s] * sy) for s in (0, 1))
        central = torch.stack([m, sum(0.5 * (m * ux[s] + p[s] * sx) for s in (0, 1)),
                               sum(0.5 * (m * uy[s] + p[s] * sy) for s in (0, 1)), sum(0.5 * m * h[s] for s in (0, 1))], 1)

        def least(l, r, lt, rt_):
            d = torch.minimum(torch.minimum((r - l).abs(), (r - lt).abs()), torch.minimum((rt_ - l).abs(), (rt_ - lt).abs()))
            return torch.where(r >= l, d, -d)

        dp, drho = least(p[0], p[1], td[0][:, 0], td[1][:, 0]), least(rho[0], rho[1], rt[0], rt[1])
        # Roe
        gam = (Cv + R) / Cv
        cv = [ux[s] * nx + uy[s] * ny for s in (0, 1)]
        sq = [torch.sqrt(r.clamp(min=1e-20)) for r in rho]
        rr = torch.sqrt((rho[0] * rho[1]).clamp(min=1e-20))
        a = sq[0] / (sq[0] + sq[1])
        mean = lambda q: q[0] * a + q[1] * (1 - a)  # noqa: E731
        uxm, uym, hm = mean(ux), mean(uy), mean(h)
        q2 = uxm ** 2 + uym ** 2
        c = torch.sqrt(((gam - 1) * (hm - 0.5 * q2)).clamp(min=1e-20))
        cs = [torch.sqrt(((gam - 1) * (h[s] - ke[s])).clamp(min=1e-20)) for s in (0, 1)]
        um = uxm * nx + uym * ny
        dux, duy = ux[1] - ux[0], uy[1] - uy[0]
        dcv = dux * nx + duy * ny
        r1, r2, r3 = (dp - rr * c * dcv) / (2 * c * c), drho - dp / (c * c), (dp + rr * c * dcv) / (2 * c * c)

        def fix(lam, jump):
            e = 2 * jump.clamp(min=0.0)
            return torch.where(lam >= e, lam, (lam * lam + e * e) / (2 * e + 1e-30))

        l1 = fix((um - c).abs(), (cv[1] - cs[1]) - (cv[0] - cs[0]))
        l2 = fix(um.abs(), cv[1] - cv[0])
        l3 = fix((um + c).abs(), (cv[1] + cs[1]) - (cv[0] + cs[0]))
        diss = torch.stack([
            l1 * r1 + l2 * r2 + l3 * r3,
            l1 * r1 * (uxm - c * nx) + l2 * (r2 * uxm + rr * (dux - dcv * nx)) + l3 * r3 * (uxm + c * nx),
            l1 * r1 * (uym - c * ny) + l2 * (r2 * uym + rr * (duy - dcv * ny)) + l3 * r3 * (uym + c * ny),
            l1 * r1 * (hm - c * um) + l2 * (r2 * 0.5 * q2 + rr * (uxm * dux + uym * duy - um * dcv))
            + l3 * r3 * (hm + c * um)], 1)
        roe = central - 0.5 * diss * mag[:, None]
        if not bool(kfvs.any()):
            return roe
        # kinetic flux-vector splitting
        mom = []
        for s, sg in ((0, 1.0), (1, -1.0)):
            lam = 0.5 * rho[s] / p[s]
            u = cv[s]
            m0 = 0.5 * torch.erfc(-sg * torch.sqrt(lam) * u)
            m1 = u * m0 + sg * 0.5 * torch.exp(-lam * u * u) / torch.sqrt(self.pi * lam)
            m2 = u * m1 + 0.5 * m0 / lam
            m3 = u * m2 + m1 / lam
            v = uy[s] * nx - ux[s] * ny
            K = 2 * Cv / R - 2
            mom.append((rho[s] * m1, rho[s] * m2, rho[s] * m1 * v,
                        0.5 * rho[s] * (m3 + m1 * (v * v + 0.5 / lam) + m1 * K * 0.5 / lam)))
        t0, t1, t2, t3 = (x + y for x, y in zip(*mom))
        kin = torch.stack([t0 * mag, t1 * sx - t2 * sy, t1 * sy + t2 * sx, t3 * mag], 1)
        return torch.where(kfvs[:, None], kin, roe)
