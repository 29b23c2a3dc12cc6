"""The work that a user of this framework has it do, as measurable cases.

A user builds the FDFD operator A = Cₘ·Cₑ − ω²·Pε of a grid, a PML and a set
of objects, applies it (the inner step of every solver, their own or the
library's), solves A x = b, differentiates through the solve, and
post-processes the fields.  The sizes and materials are those of
``workloads.py`` and of the tests: grids of 48³ … 320³ cells, 8- to 12-cell
PML, dielectric spheres of ε = 2.25 or 12.25 with smoothed interfaces.

Field vectors are DOF vectors, component fastest, as (3·Ncell, 2) real tensors
on the GPU (float32 for complex64, float64 for complex128).
"""
import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The framework (its folder's name is not a Python identifier)."""
    name = "maxwellfdm_gb300"
    if name not in sys.modules:
        folder = os.path.join(_ROOT, "maxwellfdm.jl_gb300")
        spec = importlib.util.spec_from_file_location(name, os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _apply(name, n, prec="c64", **kw):
    c = {"name": name, "kind": "apply", "nx": n[0], "ny": n[1], "nz": n[2], "prec": prec, "ft": "E", "bloch": "",
         "pml": 10, "lam": 16.0, "spheres": 0, "rlo": 3.0, "rhi": 8.0, "eps": 12.25}
    c.update(kw)
    return c


def listed():
    return [
        # one application in a user's own Krylov loop on the smallest grid of the uneven batch: launch and latency count
        _apply("apply_c64_48", (48, 48, 48), pml=8, spheres=10),
        # the sphere scatterer that bench.py solves: the inner step of its mixed-precision solve
        _apply("apply_c64_96", (96, 96, 96), spheres=40),
        # the largest configuration, streamed from HBM
        _apply("apply_c64_320", (320, 320, 320), pml=12, lam=24.0, spheres=400, rlo=4.0, rhi=16.0),
        # a grid nobody rounded: every extent odd, no multiple of a tile
        _apply("apply_c64_odd", (95, 89, 83), spheres=30),
        # the operator in double precision (true residuals, FP64 solves), ragged in every axis
        _apply("apply_c128_ragged", (110, 90, 77), "c128", spheres=30),
        # a periodic cell (photonic crystal, metasurface) at a Bloch vector: periodic in x and y, PML in z
        _apply("apply_bloch_c64", (64, 64, 96), bloch="xy", spheres=12, rhi=6.0),
        # the H formulation (diagonal ε), inner step of its solve
        _apply("apply_h_c64", (96, 96, 96), ft="H", spheres=20),
        # after a solve: H from E, and both fields averaged to voxel corners, on the inverse-design grid
        {"name": "fields_c128", "kind": "fields", "nx": 128, "ny": 128, "nz": 64, "bloch": "", "pml": 10, "lam": 16.0},
        # geometry update: objects moved, ε assigned and smoothed again, then one FP64 application
        {"name": "smooth_96", "kind": "smooth", "nx": 96, "ny": 96, "nz": 96, "pml": 10, "lam": 16.0, "spheres": 40,
         "rlo": 3.0, "rhi": 8.0, "eps": 12.25},
        # the vacuum dipole box in plain FP64, host arrays in and out (the plain method)
        {"name": "solve_fp64_32", "kind": "solve", "nx": 32, "ny": 32, "nz": 32, "prec": "fp64", "pml": 10, "lam": 20.0,
         "spheres": 0, "rlo": 3.0, "rhi": 4.0, "eps": 2.25, "host": True, "apps": 586},
        # a scatterer of low-index spheres in mixed precision, device buffers: the solver's own kernels at full size
        {"name": "solve_mixed_96", "kind": "solve", "nx": 96, "ny": 96, "nz": 96, "prec": "mixed", "pml": 10, "lam": 16.0,
         "spheres": 40, "rlo": 3.0, "rhi": 8.0, "eps": 2.25, "host": False, "apps": 3608},
        # inverse design: the adjoint solve of a slab waveguide and the gradient at every sample, host arrays
        {"name": "grad_mixed_slab", "kind": "grad", "nx": 64, "ny": 64, "nz": 32, "prec": "mixed", "pml": 8, "lam": 16.0,
         "apps": 2348},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def edges(lo, hi):
        return {"nx": logint(lo, hi), "ny": logint(lo, hi), "nz": logint(lo, hi)}

    kind = rng.choice(["apply", "apply", "apply", "bloch", "h", "fields", "smooth", "solve"])
    c = {"pml": rng.choice([8, 10]), "lam": round(rng.uniform(12.0, 24.0), 3)}
    if kind in ("apply", "bloch", "h"):
        c = dict(_apply("", (1, 1, 1)), **c)
        del c["name"]
        c.update(edges(32, 256))
        c["prec"] = rng.choice(["c64", "c64", "c128"])
        c["spheres"] = max(1, min(200, c["nx"] * c["ny"] * c["nz"] // 30000)) if rng.random() < 0.8 else 0
        if kind == "bloch":
            c["bloch"] = rng.choice(["x", "xy", "z", "xyz", "slab"])
            if c["bloch"] == "slab":  # a 2D model: one periodic cell along z
                c.update(bloch="z", nx=logint(64, 1024), ny=logint(64, 1024), nz=1, spheres=0)
        elif kind == "h":
            c["ft"] = "H"
    elif kind == "fields":
        c.update(edges(32, 200), kind="fields", bloch=rng.choice(["", "", "xy", "z"]))
    elif kind == "smooth":
        c.update(edges(48, 160), kind="smooth", rlo=3.0, rhi=8.0, eps=rng.choice([2.25, 12.25]))
        c["spheres"] = max(4, min(60, c["nx"] * c["ny"] * c["nz"] // 25000))
    else:
        c.update(edges(28, 56), kind="solve", prec=rng.choice(["fp64", "mixed"]), spheres=rng.randint(0, 3), rlo=2.0,
                 rhi=4.0, eps=2.25, host=rng.random() < 0.5, apps=600)
    return c


# ------------------------------------------------------------------ inputs
def _bloch(case):
    return tuple(a in case.get("bloch", "") for a in "xyz")


def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _phases(case, rng):
    """e^{−i k L} per axis: a Bloch vector in the first zone (a 2D slice has none along z)."""
    out = []
    for n, b in zip(_dims(case), _bloch(case)):
        k = rng.uniform(-1.0, 1.0)
        out.append(complex(np.exp(-1j * math.pi * k)) if b and n > 1 else 1.0 + 0.0j)
    return tuple(out)


def _omega(case):
    return 2 * math.pi / case["lam"]


def _stretched(case):
    """(s∆lₑ, s∆lₘ) of unit cells with the usual polynomial PML (m = 4, R = 1e-8) on every axis that is not periodic."""
    om, se, sm = _omega(case), [], []
    for n, b in zip(_dims(case), _bloch(case)):
        p = 0 if b else min(case["pml"], (n - 4) // 2)
        both = []
        for u in (np.arange(n) * 1.0, np.arange(n) + 0.5):
            sig = np.zeros(n)
            if p > 0:
                depth = np.maximum(0.0, np.maximum(p - u, u - (n - p)))
                sig = -(5.0 * math.log(1e-8)) / (2.0 * p) * (depth / p) ** 4
            both.append(1.0 + sig / (1j * om))
        se.append(both[0])
        sm.append(both[1])
    return se, sm


def _sphere_list(case, rng):
    """Non-overlapping spheres inside the PML, at least two cells apart: (centre, radius) rows."""
    n = np.array(_dims(case), dtype=float)
    lo = np.where(_bloch(case), 0.0, np.minimum(case["pml"], (n - 4) // 2))
    hi = n - lo
    got = np.zeros((0, 4))
    for _ in range(200 * max(1, case["spheres"])):
        if len(got) >= case["spheres"]:
            break
        r = rng.uniform(case["rlo"], case["rhi"])
        if np.any(hi - lo <= 2 * r + 1):
            continue
        c = rng.uniform(lo + r, hi - r)
        if len(got) == 0 or np.all(np.linalg.norm(got[:, :3] - c, axis=1) > r + got[:, 3] + 2.0):
            got = np.vstack([got, np.append(c, r)])
    return got


def _eps(case, rng):
    """ε as such a program has it: (diagonal at the E samples, off-diagonal xy, yz, zx at the voxel corners), as
    (Nz, Ny, Nx, 3) float64 on the GPU.  Interfaces carry the smoothed tensor ε̃ = ⟨ε⟩ I + (⟨ε⁻¹⟩⁻¹ − ⟨ε⟩) n nᵀ with the fill of
    the plane through the voxel taken from the signed distance."""
    nx, ny, nz = _dims(case)
    diag = torch.ones(nz, ny, nx, 3, dtype=torch.float64, device="cuda")
    off = torch.zeros_like(diag)
    for cx, cy, cz, r in _sphere_list(case, rng):
        a = [max(0, int(math.floor(c - r)) - 2) for c in (cx, cy, cz)]
        b = [min(n, int(math.ceil(c + r)) + 3) for c, n in zip((cx, cy, cz), (nx, ny, nz))]
        ax = [torch.arange(a[w], b[w], dtype=torch.float64, device="cuda") for w in range(3)]
        box = (slice(a[2], b[2]), slice(a[1], b[1]), slice(a[0], b[0]))
        for s in range(4):  # E_x, E_y, E_z samples, corners
            d = [ax[w] + (0.5 if w == s else 0.0) - (cx, cy, cz)[w] for w in range(3)]
            dx, dy, dz = d[0][None, None, :], d[1][None, :, None], d[2][:, None, None]
            dist = torch.sqrt(dx * dx + dy * dy + dz * dz).clamp_min(1e-12)
            fill = (0.5 + (r - dist)).clamp(0.0, 1.0)
            mean = 1.0 + fill * (case["eps"] - 1.0)
            harm = 1.0 / (1.0 + fill * (1.0 / case["eps"] - 1.0))
            if s < 3:
                nrm = (dx, dy, dz)[s] / dist
                diag[box + (s,)] = torch.where(fill > 0, mean + (harm - mean) * nrm * nrm, diag[box + (s,)])
            else:
                for p, (u, v) in enumerate(((dx, dy), (dy, dz), (dz, dx))):
                    off[box + (p,)] = torch.where(fill > 0, (harm - mean) * (u * v) / (dist * dist), off[box + (p,)])
    return diag, off


def _vector(case, gen, n=None, dtype=torch.float64):
    """A seeded complex Gaussian DOF vector."""
    nx, ny, nz = _dims(case)
    return torch.randn(n or 3 * nx * ny * nz, 2, generator=gen, device="cuda", dtype=dtype)


def _material(case, rng):
    diag, off = _eps(case, rng) if case["spheres"] else (None, None)
    if diag is not None and case["ft"] == "H":
        off = None  # the H formulation takes a diagonal ε
    if off is not None and not bool((off != 0).any()):
        off = None
    return diag, off


def _operator(case, phases):
    pkg = _package()
    se, sm = _stretched(case)
    return pkg.FDFDOperator(_dims(case), _omega(case), se, sm, _bloch(case), phases)


def _host_cells(a):
    return None if a is None else a.cpu().numpy().transpose(2, 1, 0, 3)


def _model(case, rng):
    pkg = _package()
    mdl = pkg.ModelFull(pkg.uniform_grid(_dims(case)))
    om = _omega(case)
    pkg.set_ωpml(mdl, om)
    p = tuple(min(case["pml"], (n - 8) // 2) for n in _dims(case))
    pkg.set_Npml(mdl, (p, p))
    if case.get("spheres"):
        for s in _sphere_list(dict(case, pml=max(p)), rng):
            pkg.add_obj(mdl, "dielectric", pkg.Sphere(s[:3], s[3]), ε=case["eps"])
    return mdl, om, p


def _streams_done():
    torch.cuda.synchronize()


def prepare(case, seed):
    pkg = _package()
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind = case["kind"]
    st = {"case": case}
    if kind == "apply":
        phases = _phases(case, rng)
        diag, off = _material(case, rng)
        A = _operator(case, phases)
        if diag is not None:
            A.set_eps(_host_cells(diag), _host_cells(off))
        del diag, off
        if case["ft"] == "H":
            A.set_field_type("H")
        st["x"] = _vector(case, gen, dtype=torch.float32 if case["prec"] == "c64" else torch.float64)
        st["y"] = torch.empty_like(st["x"])
    elif kind == "fields":
        A = _operator(case, _phases(case, rng))
        st["e"], st["jm"] = _vector(case, gen), _vector(case, gen)
        st["h"], st["ec"], st["hc"] = (torch.empty_like(st["e"]) for _ in range(3))
    elif kind == "smooth":
        mdl, om, _ = _model(case, rng)
        A = pkg.create_A(mdl, om)
        moved, _, _ = _model(case, rng)  # the next geometry of the same program
        st["lprim"], st["objects"] = mdl.grid.lprim, moved.objects
        st["x"] = _vector(case, gen)
        st["y"] = torch.empty_like(st["x"])
    elif kind == "solve":
        mdl, om, p = _model(case, rng)
        n = np.array(_dims(case), dtype=float)
        at = rng.uniform(np.array(p) + 2.0, n - np.array(p) - 2.0)
        pol = rng.standard_normal(3)
        pkg.add_srce(mdl, pkg.PointSrc(at, pol / np.linalg.norm(pol)))
        A, b = pkg.create_linsys(mdl, om)
        if case["host"]:
            st["b"] = b
        else:
            st["b"] = torch.from_numpy(b.view(np.float64).reshape(-1, 2).copy()).cuda()
            st["x"] = torch.zeros_like(st["b"])
    else:  # grad: a slab waveguide, the objective a Gaussian mode profile on an output plane
        mdl, om, p = _model(case, rng)
        nx, ny, nz = _dims(case)
        pkg.add_obj(mdl, "slab", pkg.Box((-1.0, -1.0, nz / 2 - 4.0), (nx + 1.0, ny + 1.0, nz / 2 + 4.0)), ε=12.25)
        pkg.set_design(mdl, pkg.DesignRegion((nx // 3, ny // 3, nz // 2 - 4), (2 * nx // 3, 2 * ny // 3, nz // 2 + 4),
                                             rng.uniform(1.0, 12.25, (2 * nx // 3 - nx // 3, 2 * ny // 3 - ny // 3, 8))))
        A = pkg.create_A(mdl, om)
        prof = np.exp(-((np.arange(ny)[:, None] + 0.5 - ny / 2 - rng.uniform(-1, 1)) ** 2
                        + (np.arange(nz)[None, :] - nz / 2) ** 2) / 72.0)
        g = np.zeros((nx, ny, nz, 3), dtype=np.complex128)
        g[nx - p[0] - 8, :, :, 1] = prof
        st["g"] = pkg.field_arr2vec(g)
        st["e"] = rng.standard_normal(A.n) + 1j * rng.standard_normal(A.n)
    st["A"] = A
    _streams_done()
    return st


# ------------------------------------------------------------------ one pass
def run(st):
    case, A = st["case"], st["A"]
    kind = case["kind"]
    if kind == "apply":
        A.matvec_dev(st["x"].data_ptr(), st["y"].data_ptr(), case["prec"])
        return st["y"]
    if kind == "fields":
        lib, h = A._lib, A._h
        e, jm, hf, ec, hc = (ctypes.c_void_p(st[k].data_ptr()) for k in ("e", "jm", "h", "ec", "hc"))
        A._check(lib.fdfd_h_from_e_dev(h, e, jm, hf))
        A._check(lib.fdfd_corner_mean_dev(h, 0, e, ec))
        A._check(lib.fdfd_corner_mean_dev(h, 1, hf, hc))
        return [st["h"], st["ec"], st["hc"]]
    if kind == "smooth":
        A.smooth_objects(st["lprim"], st["objects"], 1.0)
        A.matvec_dev(st["x"].data_ptr(), st["y"].data_ptr(), "c128")
        return st["y"]
    # solutions to a 1e-12 true residual: fields that two programs can compare
    if kind == "solve":
        if case["host"]:
            return A.solve(st["b"], tol=1e-12, precision=case["prec"])[0]
        A.solve_dev(st["b"].data_ptr(), st["x"].data_ptr(), tol=1e-12, precision=case["prec"])
        return st["x"]
    return A.eps_grad(st["e"], st["g"], tol=1e-11, precision=case["prec"])[0]


def work(case):
    """Bytes: every vector and the ε diagonal once per application; a solve or a gradient needs `apps` applications (BiCGStab(4) as measured on
    these systems).  Operations: two curls and the ε term, complex."""
    cells = case["nx"] * case["ny"] * case["nz"]
    kind = case["kind"]
    if kind == "apply":
        return {"bytes": cells * (60 if case["prec"] == "c64" else 120), "flops": cells * 100}
    if kind == "fields":
        return {"bytes": cells * (144 + 96 + 96), "flops": cells * 150}
    if kind == "smooth":  # ε written (diagonal and off-diagonal), then one application
        return {"bytes": cells * (48 + 120), "flops": cells * 100}
    return {"bytes": cells * case["apps"] * (120 if case["prec"] == "fp64" else 60), "flops": cells * case["apps"] * 100}


# ------------------------------------------------------------------ the same in 64 bits, in plain torch
class _Grid:
    """Difference and averaging operators on (Nz, Ny, Nx) complex128 fields (axis 0, 1, 2 = x, y, z here)."""

    def __init__(self, case, phases):
        self.bloch, self.ph = _bloch(case), phases
        se, sm = _stretched(case)
        self.se = [torch.from_numpy(v).cuda() for v in se]
        self.sm = [torch.from_numpy(v).cuda() for v in sm]
        nx, ny, nz = _dims(case)
        self.first = []
        for w, n in enumerate((nx, ny, nz)):
            m = torch.zeros(n, dtype=torch.bool, device="cuda")
            m[0] = not self.bloch[w]
            self.first.append(self.along(m, w))

    @staticmethod
    def along(v, w):
        return v.reshape([-1 if d == 2 - w else 1 for d in range(3)])

    def nxt(self, f, w):
        """f at index + 1 along w; beyond the end 0, or the periodic image."""
        g = torch.roll(f, -1, 2 - w)
        last = g.narrow(2 - w, f.shape[2 - w] - 1, 1)
        last.mul_(self.ph[w] if self.bloch[w] else 0.0)
        return g

    def prv(self, f, w, mirror):
        """f at index − 1 along w; before the start f[0] (mirror) or 0, or the periodic image."""
        g = torch.roll(f, 1, 2 - w)
        at0 = g.narrow(2 - w, 0, 1)
        if self.bloch[w]:
            at0.mul_(1.0 / self.ph[w])
        elif mirror:
            at0.copy_(f.narrow(2 - w, 0, 1))
        else:
            at0.zero_()
        return g

    def pinned(self, c):
        m = torch.zeros((), dtype=torch.bool, device="cuda")
        for w in range(3):
            if w != c:
                m = m | self.first[w]
        return m

    def free(self, f):
        return [torch.where(self.pinned(c), torch.zeros((), dtype=f[c].dtype, device="cuda"), f[c]) for c in range(3)]

    def curl_e(self, f):
        d = lambda c, w: (self.nxt(f[c], w) - f[c]) / self.along(self.sm[w], w)  # noqa: E731
        return [d(2, 1) - d(1, 2), d(0, 2) - d(2, 0), d(1, 0) - d(0, 1)]

    def curl_h(self, f):
        d = lambda c, w: (f[c] - self.prv(f[c], w, True)) / self.along(self.se[w], w)  # noqa: E731
        return self.free([d(2, 1) - d(1, 2), d(0, 2) - d(2, 0), d(1, 0) - d(0, 1)])

    def corner_e(self, f, c):
        """E_c averaged backward along c onto the voxel corner."""
        w = self.along(self.sm[c], c)
        wf = w * f
        return (self.prv(wf, c, True) + wf) / (2 * self.along(self.se[c], c))

    def corner_h(self, f, c):
        wf = self.along(self.se[c], c) * f
        return (wf + self.nxt(wf, c)) / (2 * self.along(self.sm[c], c))

    def off_term(self, f, off):
        """Off-diagonal ε: corner products averaged back onto the E samples."""
        xy, yz, zx = off[..., 0], off[..., 1], off[..., 2]
        a = [self.corner_e(f[c], c) for c in range(3)]
        t = [xy * a[1] + zx * a[2], xy * a[0] + yz * a[2], zx * a[0] + yz * a[1]]
        return self.free([0.5 * (t[c] + self.nxt(t[c], c)) for c in range(3)])


def _unpack(v, case):
    nx, ny, nz = _dims(case)
    c = torch.view_as_complex(v.double().contiguous()).reshape(nz, ny, nx, 3)
    return [c[..., k].contiguous() for k in range(3)]


def _pack(f):
    return torch.view_as_real(torch.stack(f, -1).reshape(-1))


def exact(case, seed):
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["kind"] == "apply":
        phases = _phases(case, rng)
        diag, off = _material(case, rng)
        x = _unpack(_vector(case, gen, dtype=torch.float32 if case["prec"] == "c64" else torch.float64), case)
        g, w2 = _Grid(case, phases), _omega(case) ** 2
        ed = [1.0, 1.0, 1.0] if diag is None else [diag[..., c] for c in range(3)]
        if case["ft"] == "H":
            e = g.curl_h(x)
            y = g.curl_e([e[c] / ed[c] for c in range(3)])
            return _pack([y[c] - w2 * x[c] for c in range(3)])
        f = g.free(x)
        y = g.curl_h(g.curl_e(f))
        y = [y[c] - w2 * (ed[c] * x[c]) for c in range(3)]
        if off is not None:
            t = g.off_term(f, off)
            y = [y[c] - w2 * t[c] for c in range(3)]
        return _pack(y)
    if case["kind"] == "fields":
        g = _Grid(case, _phases(case, rng))
        e, jm = _unpack(_vector(case, gen), case), _unpack(_vector(case, gen), case)
        h = g.curl_e(g.free(e))
        h = [(1j / _omega(case)) * (h[c] + jm[c]) for c in range(3)]
        return [_pack(h), _pack([g.corner_e(e[c], c) for c in range(3)]), _pack([g.corner_h(h[c], c) for c in range(3)])]
    # a smoothed geometry needs the exact cut volumes, a solve or a gradient a sparse factorisation: beyond plain torch here
    return None
