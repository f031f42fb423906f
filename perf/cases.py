"""Timed cases: what users of the retarded BEM path have the library do.

Each case goes through the package's public entry points (``bemsolver``,
``planewave``, ``dipoleret``, ``meshfield``, ``spectrum_batch``,
``autograd.extinction``).  The kinds:

  sweep     a spectrum: extinction and scattering over a wavelength grid
  solve     one wavelength with the surface charges and currents (``bem \\ exc``)
  batch     the sweeps of three particles of uneven size in one call
  gradient  adjoint gradient of the extinction for a particle the user keeps
  shape     one step of a shape optimisation: new vertices, forward, backward
  map       near-field map of a solution on a grid of points
  decay     decay rates of dipoles near a particle: potentials, solve, rates
  iter      one wavelength with the H-matrix iterative solver

A seed changes the sizes by a few per cent, the metal, the wavelengths, gaps,
points and dipole positions.  ``exact`` restates the boundary element method
in 64-bit torch: geometry, refined near elements, the Garcia de Abajo - Howie
solve, cross sections, fields and (by automatic differentiation) gradients.
"""
import math
import os

import numpy as np
import torch

import mnpbem_gb300 as m
from mnpbem_gb300 import autograd, shapes

NM_PER_EV = 1.0 / 8.0655477e-4      # wavelength (nm) times photon energy (eV)
EPS_OUT = 1.77                      # water

# face counts behind the mesh parameters: rod (nphi - 1)(2 (ntheta - 1) + nz - 1)
# quadrilaterals, cube 6 (n - 1)^2


def listed():
    return [
        # smallest call: one wavelength of the 284-face gold sphere of the first
        # plane-wave demo; latency and launches count
        {"name": "solve_sphere284", "kind": "solve", "shape": "sphere", "faces": 284, "size": 150.0, "npol": 1,
         "nw": 1, "lo": 400.0, "hi": 900.0, "precision": "mixed", "curved": False},
        # that demo itself: curved elements, 40 wavelengths, two polarisations
        {"name": "sweep_sphere284_curv", "kind": "sweep", "shape": "sphere", "faces": 284, "size": 150.0, "npol": 2,
         "nw": 40, "lo": 400.0, "hi": 900.0, "precision": "mixed", "curved": True},
        # full double precision: a rounded cube of 1350 quadrilaterals
        {"name": "sweep_cube1350_fp64", "kind": "sweep", "shape": "cube", "m": 16, "size": 40.0, "npol": 2, "nw": 2,
         "lo": 500.0, "hi": 700.0, "precision": "fp64", "curved": False},
        # the single-particle benchmark: 4000-face sphere, wavelength sweep
        {"name": "sweep_sphere4000", "kind": "sweep", "shape": "sphere", "faces": 4000, "size": 50.0, "npol": 1,
         "nw": 16, "lo": 450.0, "hi": 750.0, "precision": "mixed", "curved": False},
        # a dimer sweep of ordinary size: two spheres in separate media, 2 nm gap
        {"name": "sweep_dimer8000", "kind": "sweep", "shape": "dimer", "faces": 8000, "size": 50.0, "npol": 1,
         "nw": 8, "lo": 500.0, "hi": 900.0, "precision": "mixed", "curved": False},
        # one wavelength of the headline problem, the 24 000-face dimer (the
        # largest: five 24 000 x 24 000 complex matrices and the residual planes)
        {"name": "solve_dimer24000", "kind": "solve", "shape": "dimer", "faces": 24000, "size": 50.0, "npol": 1,
         "nw": 1, "lo": 500.0, "hi": 900.0, "precision": "mixed", "curved": False},
        # the batch benchmark's particles (sphere 1000, rod 2500, cube 2904 faces)
        {"name": "batch_1000_2500_2904", "kind": "batch", "faces": 1000, "nphi": 51, "nth": 11, "nz": 31, "m": 23,
         "npol": 2, "nw": 8, "lo": 400.0, "hi": 900.0, "precision": "mixed"},
        # sensitivity of a rod's extinction, adjoint in mixed precision
        {"name": "gradient_rod2016", "kind": "gradient", "shape": "rod", "nphi": 25, "nth": 7, "nz": 31,
         "tri": True, "size": 10.0, "precision": "mixed"},
        # shape optimisation step through torch.autograd: set-up, solve, adjoint (FP64)
        {"name": "shape_sphere508", "kind": "shape", "shape": "sphere", "faces": 508, "size": 50.0},
        # near-field map around the rod with quadrilaterals, ragged point count
        {"name": "map_rod1176", "kind": "map", "shape": "rod", "nphi": 43, "nth": 8, "nz": 15, "tri": False,
         "size": 10.0, "npol": 2, "nx": 97, "nz_pts": 101, "precision": "mixed"},
        # decay rates of three dipoles with three orientations each at a sphere
        {"name": "decay_sphere1148", "kind": "decay", "shape": "sphere", "faces": 1148, "size": 50.0, "npt": 3,
         "precision": "mixed"},
        # H-matrix iterative solver on a dimer, dense preconditioner
        {"name": "iter_dimer6000", "kind": "iter", "shape": "dimer", "faces": 6000, "size": 50.0, "npol": 1,
         "precision": "mixed"},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _even(x):
    return 2 * int(round(x / 2))


def _rod(rng, lo, hi):
    """Mesh parameters of a rod with about lo..hi quadrilaterals."""
    nf = _log(rng, lo, hi)
    nphi = max(9, int(round(math.sqrt(nf) * rng.uniform(0.8, 1.2))) + 1)
    rows = max(6, int(round(nf / (nphi - 1))))
    nth = max(3, rows // 4 + rng.randrange(0, 2))
    return {"nphi": nphi, "nth": nth, "nz": max(2, rows - 2 * (nth - 1) + 1)}


def _any_shape(rng, lo, hi):
    pick = rng.random()
    if pick < 0.45:
        return {"shape": "sphere", "faces": _even(_log(rng, lo, hi)), "size": round(rng.uniform(20.0, 120.0), 1)}
    if pick < 0.75:
        return {"shape": "rod", "tri": False, "size": round(rng.uniform(8.0, 16.0), 1), **_rod(rng, lo, hi)}
    return {"shape": "cube", "m": max(4, int(round(math.sqrt(_log(rng, lo, hi) / 6))) + 1),
            "size": round(rng.uniform(20.0, 60.0), 1)}


def draw(rng):
    kind = rng.choice(["sweep", "sweep", "sweep", "solve", "dimer", "fp64", "batch", "gradient", "shape", "map",
                       "decay", "iter"])
    band = {"npol": rng.choice([1, 1, 2]), "lo": round(rng.uniform(420.0, 520.0), 1),
            "hi": round(rng.uniform(650.0, 900.0), 1)}
    if kind == "sweep":
        s = _any_shape(rng, 120, 4000)
        nw = int(_log(rng, 2, 40 if _faces(s) < 1500 else 14))
        return {"kind": "sweep", **s, **band, "nw": nw, "precision": "mixed",
                "curved": s["shape"] == "sphere" and s["faces"] < 2000 and rng.random() < 0.3}
    if kind == "solve":
        return {"kind": "solve", **_any_shape(rng, 120, 8000), **band, "nw": 1, "precision": "mixed", "curved": False}
    if kind == "dimer":
        nf = 2 * _even(_log(rng, 700, 6000))
        return {"kind": "sweep", "shape": "dimer", "faces": nf, "size": 50.0, **band,
                "nw": rng.randrange(2, 9 if nf < 6000 else 5), "precision": "mixed", "curved": False}
    if kind == "fp64":
        return {"kind": "sweep", **_any_shape(rng, 120, 1400), **band, "nw": rng.randrange(1, 4), "precision": "fp64",
                "curved": False}
    if kind == "batch":
        return {"kind": "batch", "faces": _even(_log(rng, 300, 1500)), **_rod(rng, 500, 2600),
                "m": rng.randrange(9, 23), "npol": rng.choice([1, 2]), "nw": rng.randrange(2, 9), "lo": 420.0,
                "hi": 880.0, "precision": "mixed"}
    if kind == "gradient":
        prec = rng.choice(["mixed", "mixed", "fp64"])
        return {"kind": "gradient", "shape": "rod", "tri": True, "size": round(rng.uniform(8.0, 14.0), 1),
                "precision": prec, **_rod(rng, 150, 1100 if prec == "mixed" else 500)}
    if kind == "shape":
        return {"kind": "shape", "shape": "sphere", "faces": _even(_log(rng, 100, 900)),
                "size": round(rng.uniform(20.0, 80.0), 1)}
    if kind == "map":
        return {"kind": "map", **_any_shape(rng, 200, 2500), "npol": rng.choice([1, 2]), "nx": rng.randrange(21, 120),
                "nz_pts": rng.randrange(21, 120), "precision": "mixed"}
    if kind == "decay":
        return {"kind": "decay", **_any_shape(rng, 200, 2000), "npt": rng.randrange(1, 5), "precision": "mixed"}
    return {"kind": "iter", "shape": "dimer", "faces": 2 * _even(_log(rng, 1000, 4000)), "size": 50.0,
            "npol": rng.choice([1, 2]), "precision": "mixed"}


# ------------------------------------------------------------------ problems
def _faces(c):
    if c["shape"] == "rod":
        return (c["nphi"] - 1) * (2 * (c["nth"] - 1) + c["nz"] - 1) * (2 if c.get("tri") else 1)
    if c["shape"] == "cube":
        return 6 * (c["m"] - 1) ** 2
    return c["faces"]


_MESH = {}


def _unit_mesh(c):
    """Mesh of the case's shape at its nominal size (a mesh file in a user's hands)."""
    key = (c["shape"], c.get("faces"), c.get("m"), c.get("nphi"), c.get("nth"), c.get("nz"), c.get("tri"), c["size"])
    if key not in _MESH:
        if c["shape"] == "rod":
            v, f = shapes.trirod(c["size"], 4 * c["size"], (c["nphi"], c["nth"], c["nz"]), triangles=c["tri"])
        elif c["shape"] == "cube":
            v, f = shapes.tricube(c["m"], c["size"], shapes.rounding_to_e(c["size"], 0.1 * c["size"]))
        else:
            v, f = shapes.sphere(c["faces"] // (2 if c["shape"] == "dimer" else 1), c["size"])
        f = np.asarray(f, dtype=np.int64)
        if f.shape[1] == 3:
            f = np.hstack([f, -np.ones((f.shape[0], 1), np.int64)])
        _MESH[key] = (np.asarray(v, dtype=np.float64), f)
    return _MESH[key]


class _Problem:
    """Meshes, media and wavelengths of a case for one seed (plain arrays)."""

    def __init__(self, case, seed):
        rng = np.random.default_rng([int(seed), 77])
        u = rng.uniform(-1.0, 1.0, 8)
        self.wp, self.gamma = 9.065 * (1 + 0.01 * u[0]), 0.0708 * (1 + 0.1 * u[1])
        self.rng = rng
        scale = 1 + 0.02 * u[2]
        v, f = _unit_mesh(case)
        v = v * scale
        self.axis_z = case["shape"] == "rod"
        self.curved = bool(case.get("curved"))
        if case["shape"] == "dimer":
            shift = 0.5 * scale * case["size"] + 1.0 + 0.1 * u[3]
            s = np.array([[shift, 0.0, 0.0]])
            self.meshes = [(v - s, f), (v + s, f)]
            self.inout = [[2, 1], [3, 1]]
        else:
            self.meshes = [(v, f)]
            self.inout = [[2, 1]]
        if self.curved:
            nodes = []
            for v, f in self.meshes:
                v2, f2 = shapes.midpoints_flat(v, f)
                r = np.sqrt(np.sum(v2 * v2, 1))[:, None]
                nodes.append((v2 * (0.5 * scale * case["size"]) / r, f2))
            self.nodes = nodes
        if "nw" in case:
            self.enei = (np.linspace(case["lo"], case["hi"], case["nw"]) if case["nw"] > 1
                         else np.array([0.5 * (case["lo"] + case["hi"])])) + 4.0 * u[4]
        else:
            self.enei = np.array([600.0 + 40.0 * u[4]])
        npol = case.get("npol", 1)
        if self.axis_z:
            self.pol, self.dir = [[0.0, 0.0, 1.0], [0.0, 1.0, 0.0]][:npol], [[1.0, 0.0, 0.0]] * npol
        else:
            self.pol, self.dir = [[1.0, 0.0, 0.0], [0.0, 1.0, 0.0]][:npol], [[0.0, 0.0, 1.0]] * npol

    def metal(self, ev):
        return 10 - self.wp ** 2 / (ev * (ev + 1j * self.gamma))

    def eps(self, enei):
        """Dielectric functions of the media at one wavelength."""
        e = complex(self.metal(NM_PER_EV / enei))
        return [complex(EPS_OUT)] + [e] * len(self.meshes)

    def comparticle(self):
        metal = m.epsfun(self.metal, "eV")
        if self.curved:
            parts = [m.particle(v, f, {"interp": "curv"}) for v, f in self.nodes]
        else:
            parts = [m.particle(v, f) for v, f in self.meshes]
        return m.comparticle([m.epsconst(EPS_OUT)] + [metal] * len(parts), parts, self.inout,
                             *range(1, len(parts) + 1))

    def points(self, case):
        """Grid through the particle, from its inside to two radii away."""
        v = self.meshes[0][0]
        lo, hi = v.min(0), v.max(0)
        mid, half = 0.5 * (lo + hi), 0.5 * (hi - lo)
        off = self.rng.uniform(-0.3, 0.3, 3)
        x = np.linspace(mid[0] - half[0] - 12.0, mid[0] + half[0] + 12.0, case["nx"]) + off[0]
        z = np.linspace(mid[2] - half[2] - 12.0, mid[2] + half[2] + 12.0, case["nz_pts"]) + off[2]
        X, Z = np.meshgrid(x, z, indexing="ij")
        return np.stack([X.ravel(), np.full(X.size, mid[1] + off[1]), Z.ravel()], 1)

    def dipoles(self, case):
        """Positions 4 to 20 nm outside the bounding sphere."""
        v = self.meshes[0][0]
        r = np.sqrt(np.sum(v * v, 1)).max()
        d = self.rng.normal(size=(case["npt"], 3))
        d /= np.sqrt(np.sum(d * d, 1))[:, None]
        return d * (r + self.rng.uniform(4.0, 20.0, case["npt"]))[:, None]


def _batch_cases(case):
    shared = {k: case[k] for k in ("npol", "nw", "lo", "hi")}
    return [{"shape": "sphere", "faces": case["faces"], "size": 30.0, **shared},
            {"shape": "rod", "tri": False, "nphi": case["nphi"], "nth": case["nth"], "nz": case["nz"], "size": 10.0,
             **shared},
            {"shape": "cube", "m": case["m"], "size": 40.0, **shared}]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        items = []
        for i, c in enumerate(_batch_cases(case)):
            p = _Problem(c, 10 * int(seed) + i)
            bem = m.bemsolver(p.comparticle(), m.bemoptions(precision=case["precision"]))
            items.append((bem, m.planewave(p.pol, p.dir), p.enei))
        return {"kind": kind, "items": items}
    p = _Problem(case, seed)
    if kind == "shape":
        v, f = p.meshes[0]
        e = p.eps(p.enei[0])[1]
        return {"kind": kind, "faces": f, "enei": float(p.enei[0]),
                "verts": torch.tensor(v, dtype=torch.float64, device="cuda"),
                "eps": torch.tensor([e.real, e.imag], dtype=torch.float64, device="cuda"), "pol": p.pol[0],
                "dir": p.dir[0]}
    cp = p.comparticle()
    op = {"precision": case["precision"]}
    if kind == "iter":
        op["iter"] = {"tol": 1e-10}                 # as tight as the direct solver's refinement
    bem = m.bemsolver(cp, m.bemoptions(**op))
    st = {"kind": kind, "bem": bem, "cp": cp, "enei": p.enei}
    if kind == "decay":
        st["pos"] = p.dipoles(case)
        st["dip"] = m.dipoleret(cp, st["pos"])
        return st
    st["exc"] = m.planewave(p.pol, p.dir)
    if kind == "gradient":
        st["precision"] = case["precision"]
    if kind == "map":
        st["mesh"] = m.meshfield(bem, p.points(case))
        st["sig"] = bem.mldivide(st["exc"](cp, float(p.enei[0])))
    return st


def run(st):
    kind = st["kind"]
    if kind == "sweep":
        r = st["bem"].spectrum(st["exc"], st["enei"])
        return {"ext": r["ext"], "sca": r["sca"]}
    if kind in ("solve", "iter"):
        s = st["bem"].mldivide(st["exc"](st["cp"], float(st["enei"][0])))
        return {k: getattr(s, k) for k in ("ext", "sca", "sig1", "sig2", "h1", "h2")}
    if kind == "batch":
        return [{"ext": r["ext"], "sca": r["sca"]} for r in m.spectrum_batch(st["items"])]
    if kind == "gradient":
        val, gv, ge = st["bem"].cross_section_gradient(st["exc"], float(st["enei"][0]), 0, "ext", st["precision"])
        return {"ext": val, "verts": gv, "eps": np.array([ge.real, ge.imag])}
    if kind == "shape":
        v, e = st["verts"].detach().requires_grad_(), st["eps"].detach().requires_grad_()
        val = autograd.extinction(v, e, st["faces"], st["enei"], st["pol"], st["dir"], EPS_OUT)
        val.backward()
        return {"ext": val.detach(), "verts": v.grad, "eps": e.grad}
    if kind == "map":
        e, h = st["mesh"](st["sig"])
        return {"e": e, "h": h}
    sig = st["bem"].mldivide(st["dip"](st["cp"], float(st["enei"][0])))
    tot, rad, _ = st["dip"].decayrate(st["bem"], sig)
    return {"tot": tot, "rad": rad, "sig2": sig.sig2}


def _solve_flops(c):
    """Real operations of the n^3 part of one wavelength: factorisations of G1
    (per particle), G2 and Sigma 8/3 n^3 each, H1 G1^-1, H2 G2^-1 and Delta^-1
    8 n^3 each."""
    n = float(_faces(c))
    n1 = n / 2 if c["shape"] == "dimer" else n
    return (n / n1) * (8 / 3 + 8) * n1 ** 3 + (8 / 3 + 8 + 8 + 8 / 3) * n ** 3


def work(case):
    kind = case["kind"]
    if kind == "batch":
        cs = _batch_cases(case)
        return {"flops": sum(c["nw"] * _solve_flops(c) for c in cs), "bytes": float(sum(48 * _faces(c) for c in cs))}
    n = float(_faces(case))
    geo = 56.0 * n                                  # vertices and face indices
    P = case.get("npol", 1)
    if kind == "sweep":
        return {"flops": case["nw"] * _solve_flops(case), "bytes": geo + 16.0 * P * case["nw"]}
    if kind == "solve":
        return {"flops": _solve_flops(case), "bytes": geo + 128.0 * n * P}
    if kind == "gradient" or kind == "shape":
        # the solve, and the derivatives of n^2 pairs of G and F (about 200 operations each)
        return {"flops": _solve_flops(case) + 400.0 * n * n, "bytes": 2 * geo}
    if kind == "map":
        # per pair: exp(ikd), G and its gradient (about 60), 8 complex columns' worth of sums per polarisation
        npts = case["nx"] * case["nz_pts"]
        return {"flops": npts * n * (60.0 + 120.0 * P), "bytes": geo + 128.0 * n * P + (24.0 + 96.0 * P) * npts}
    if kind == "decay":
        return {"flops": _solve_flops(case), "bytes": geo + 3 * case["npt"] * 256.0 * n}
    # iterative solve with a preconditioner as dense factors
    return {"flops": _solve_flops(case), "bytes": geo + 128.0 * n * P}


# --------------------------------------------------------------- 64-bit check
TWO_PI = 2 * math.pi
ORDER, CUTOFF = 5, 3.0


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _rule18():
    t = np.load(os.path.join(os.path.dirname(os.path.abspath(m.__file__)), "data", "tables.npz"))
    return t["rule18_x"], t["rule18_y"], t["rule18_w"]


def _lobatto(n):
    """Legendre-Gauss-Lobatto nodes in decreasing order and weights (n + 1 points)."""
    P = np.polynomial.legendre.Legendre.basis(n)
    x = np.sort(np.concatenate([[-1.0, 1.0], np.real(P.deriv().roots())]))[::-1].copy()
    for _ in range(3):                              # polish the interior roots
        i = slice(1, -1)
        x[i] = x[i] - P.deriv()(x[i]) / P.deriv(2)(x[i])
    return x, 2.0 / (n * (n + 1) * P(x) ** 2)


def _polar(quad):
    """Polar rule around the centroid: 8 radial x 6 angular points per sector."""
    xr, wr = _lobatto(7)
    xa, wa = _lobatto(5)
    rho = 0.5 * (xr + 1 + 1e-6)
    if quad:
        phi, step, nsec = (90 + 45 * xa) / 180 * np.pi, 0.5 * np.pi, 4
        reach = 1 / np.abs(np.sin(phi))
    else:
        phi, step, nsec = (270 + 60 * xa) / 180 * np.pi, 2 * np.pi / 3, 3
        reach = 1 / np.abs(2 * np.sin(phi))
    X, Y, W = [], [], []
    for s in range(nsec):
        r = rho[:, None] * reach[None, :]
        X.append((r * np.cos(phi + s * step)[None, :]).ravel())
        Y.append((r * np.sin(phi + s * step)[None, :]).ravel())
        W.append((wr[:, None] * wa[None, :] * rho[:, None] * reach[None, :] ** 2).ravel())
    X, Y, W = np.concatenate(X), np.concatenate(Y), np.concatenate(W)
    if quad:
        return X, Y, 4 * W / W.sum()
    return (1 - math.sqrt(3) * X - Y) / 3, (1 + math.sqrt(3) * X - Y) / 3, W / W.sum()


def _tri6(x, y):
    z = 1 - x - y
    s = np.stack([x * (2 * x - 1), y * (2 * y - 1), z * (2 * z - 1), 4 * x * y, 4 * y * z, 4 * z * x], 1)
    sx = np.stack([4 * x - 1, 0 * y, 1 - 4 * z, 4 * y, -4 * y, 4 * (z - x)], 1)
    sy = np.stack([0 * x, 4 * y - 1, 1 - 4 * z, 4 * x, 4 * (z - y), -4 * x], 1)
    return s, sx, sy


def _unit(a):
    return a / a.square().sum(-1, keepdim=True).sqrt()


def _split(z):
    return z.real, z.imag


class _Reference:
    """The boundary element method of the retarded solver in 64-bit torch."""

    def __init__(self, meshes, inout, verts=None, curved=False):
        dev = self.dev = _dev()
        T = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
        self.T = T
        off, fs, vs = 0, [], []
        for v, f in meshes:
            f = f.copy()
            f[f >= 0] += off
            off += v.shape[0]
            fs.append(f)
            vs.append(v)
        F, V = np.vstack(fs), np.vstack(vs)
        self.sizes = [f.shape[0] for _, f in meshes]
        self.inout = inout
        n = self.n = F.shape[0]
        self.v = T(V) if verts is None else verts
        med = np.repeat(np.asarray(inout), self.sizes, axis=0)
        self.med = torch.as_tensor(med, device=dev)
        (self._curved if curved else self._flat)(V, F)
        rad = torch.zeros(n, dtype=torch.float64, device=dev)
        with torch.no_grad():
            for c in range(4):
                ok = torch.as_tensor(F[:, c] >= 0, device=dev)
                d = (self.v[torch.as_tensor(np.maximum(F[:, c], 0), device=dev)] - self.pos).square().sum(1).sqrt()
                rad = torch.where(ok, torch.maximum(rad, d), rad)
            self.rad = rad
            p = self.pos
            sq = p.square().sum(1)
            d2 = sq[:, None] + sq[None, :] - 2 * p @ p.T
            d = torch.where(d2 < 1e-10, torch.zeros_like(d2), d2).clamp_min(0).sqrt()
            near = ((d - rad[None, :]) / rad[:, None] < CUTOFF) & (d != 0)
            near.fill_diagonal_(False)
            self.ri, self.rj = near.nonzero(as_tuple=True)
            del d2, d, near
        self._coefficients()

    # geometry: centroids, areas, normals, tangents, points of the two rules
    def _flat(self, V, F):
        T, v, n, dev = self.T, self.v, self.n, self.dev
        q4 = F[:, 3] >= 0
        quad = torch.as_tensor(q4, device=dev)
        c = [v[torch.as_tensor(np.where(F[:, k] >= 0, F[:, k], F[:, 0]), device=dev)] for k in range(4)]
        self.pos = torch.where(quad[:, None], (c[0] + c[1] + c[2] + c[3]) / 4, (c[0] + c[1] + c[2]) / 3)

        def tri_np(a, b, d):          # area with separately rounded operations: decides ties between halves
            x, y = V[a] - V[b], V[d] - V[b]
            N = np.stack([x[:, 1] * y[:, 2] - x[:, 2] * y[:, 1], x[:, 2] * y[:, 0] - x[:, 0] * y[:, 2],
                          x[:, 0] * y[:, 1] - x[:, 1] * y[:, 0]], 1)
            return 0.5 * np.sqrt(N[:, 0] * N[:, 0] + N[:, 1] * N[:, 1] + N[:, 2] * N[:, 2])
        F3 = np.where(F[:, 3] >= 0, F[:, 3], F[:, 0])
        second = torch.as_tensor(q4 & (tri_np(F[:, 2], F3, F[:, 0]) > tri_np(F[:, 0], F[:, 1], F[:, 2])), device=dev)

        def basis(a, b, d):
            x, y = a - b, d - b
            N = torch.linalg.cross(x, y)
            ar = 0.5 * N.square().sum(1).sqrt()
            return N, x, ar
        N1, x1, a1 = basis(c[0], c[1], c[2])
        N2, x2, a2 = basis(c[2], torch.where(quad[:, None], c[3], c[1]), torch.where(quad[:, None], c[0], c[0]))
        self.area = a1 + torch.where(quad, a2, torch.zeros_like(a2))
        self.nvec = _unit(torch.where(second[:, None], N2, N1))
        self.t1 = _unit(torch.where(second[:, None], x2, x1))
        self.t2 = torch.linalg.cross(self.nvec, self.t1)
        x, y, w = _rule18()
        S = T(np.stack([x, y, 1 - x - y], 1))
        w = T(w)
        pa = torch.einsum("pk,knc->npc", S, torch.stack([c[0], c[1], c[2]]))
        wa = a1[:, None] * w[None, :]
        if q4.any():
            pb = torch.einsum("pk,knc->npc", S, torch.stack([c[2], torch.where(quad[:, None], c[3], c[1]), c[0]]))
            wb = torch.where(quad, a2, torch.zeros_like(a2))[:, None] * w[None, :]
            pb = torch.where(quad[:, None, None], pb, pa)
            pa, wa = torch.cat([pa, pb], 1), torch.cat([wa, wb], 1)
        self.qp, self.qw = pa, wa
        self.polar = []
        i3, i4 = np.nonzero(~q4)[0], np.nonzero(q4)[0]
        if i3.size:
            x, y, w = _polar(False)
            i = torch.as_tensor(i3, device=dev)
            S = T(np.stack([x, y, 1 - x - y], 1))
            self.polar.append((i, torch.einsum("pk,knc->npc", S, torch.stack([c[0][i], c[1][i], c[2][i]])),
                               self.area[i][:, None] * T(w)[None, :]))
        if i4.size:
            x, y, w = _polar(True)
            i = torch.as_tensor(i4, device=dev)
            C = torch.stack([a[i] for a in c])
            S = T(0.25 * np.stack([(1 - x) * (1 - y), (1 + x) * (1 - y), (1 + x) * (1 + y), (1 - x) * (1 + y)], 1))
            Sx = T(0.25 * np.stack([-(1 - y), 1 - y, 1 + y, -(1 + y)], 1))
            Sy = T(0.25 * np.stack([-(1 - x), -(1 + x), 1 + x, 1 - x], 1))
            J = torch.linalg.cross(torch.einsum("pk,knc->npc", Sx, C), torch.einsum("pk,knc->npc", Sy, C))
            self.polar.append((i, torch.einsum("pk,knc->npc", S, C), T(w)[None, :] * J.square().sum(2).sqrt()))

    def _curved(self, V, F):
        """Six-node triangles: F [n, 9] with the edge nodes in columns 4 to 6."""
        T, dev = self.T, self.dev
        c = torch.stack([self.v[torch.as_tensor(F[:, k], device=dev)] for k in (0, 1, 2, 4, 5, 6)])
        ev = lambda S: torch.einsum("pk,knc->npc", T(S), c)

        def rule(x, y, w):
            s, sx, sy = _tri6(x, y)
            J = torch.linalg.cross(ev(sx), ev(sy))
            return ev(s), 0.5 * T(w)[None, :] * J.square().sum(2).sqrt()
        self.qp, self.qw = rule(*_rule18())
        self.area = self.qw.sum(1)
        s, sx, sy = _tri6(np.array([1 / 3]), np.array([1 / 3]))
        self.pos = ev(s)[:, 0]
        a, b = ev(sy)[:, 0], ev(sx)[:, 0]
        self.nvec, self.t1 = _unit(torch.linalg.cross(a, b)), _unit(a)
        self.t2 = torch.linalg.cross(self.nvec, self.t1)
        i = torch.arange(self.n, device=dev)
        self.polar = [(i, *rule(*_polar(False)))]

    # Taylor coefficients of the self and near elements, closed-surface rule
    def _coefficients(self):
        n, dev = self.n, self.dev
        fact = [math.factorial(o) for o in range(ORDER + 1)]
        g0 = torch.zeros(n, ORDER + 1, dtype=torch.float64, device=dev)
        f0 = torch.zeros(n, 3, ORDER + 1, dtype=torch.float64, device=dev)
        rmax = max(float((self.pos[i][:, None] - p).detach().square().sum(2).max()) for i, p, _ in self.polar) ** 0.5
        for i, p, w in self.polar:
            vec = self.pos[i][:, None] - p
            r = vec.square().sum(2).sqrt()
            rr = torch.clamp(r, min=1e-4 * rmax)
            dots = [torch.einsum("npc,nc->np", vec, b[i]) for b in (self.nvec, self.t1, self.t2)]
            g0 = g0.index_copy(0, i, torch.stack([(w * r ** (o - 1)).sum(1) / fact[o] for o in range(ORDER + 1)], 1))
            f = []
            for o in range(ORDER + 1):
                fn = ((o - 1) * w * dots[0] * r ** (o - 3)).sum(1) / fact[o]
                fa = ((o - 1) * w * dots[1] * r ** o / rr ** 3).sum(1) / fact[o]
                fb = ((o - 1) * w * dots[2] * r ** o / rr ** 3).sum(1) / fact[o]
                f.append(self.nvec[i] * fn[:, None] + self.t1[i] * fa[:, None] + self.t2[i] * fb[:, None])
            f0 = f0.index_copy(0, i, torch.stack(f, 2))
        self.g0, self.f0n = g0, torch.einsum("nco,nc->no", f0, self.nvec)
        g, f = self.pair_coefficients(self.pos[self.ri], self.rj)
        self.gp, self.fpn = g, torch.einsum("mco,mc->mo", f, self.nvec[self.ri])
        # sum of A_i F_ij over a closed particle is -2 pi A_j
        o0 = 0
        add = []
        for s in self.sizes:
            sl = slice(o0, o0 + s)
            _, Fm = self.block(sl, sl, None)
            add.append(-TWO_PI - (self.area[sl][:, None] * Fm).sum(0) / self.area[sl])
            o0 += s
        self.f0n = torch.cat([self.f0n[:, :1] + torch.cat(add)[:, None], self.f0n[:, 1:]], 1)

    def pair_coefficients(self, pts, face):
        gs, fs = [], []
        fact = [math.factorial(o) for o in range(ORDER + 1)]
        for s in range(0, max(1, pts.shape[0]), 200000):
            x, j = pts[s:s + 200000], face[s:s + 200000]
            vec = x[:, None, :] - self.qp[j]
            w = self.qw[j]
            r = vec.square().sum(2).sqrt()
            dr = r - (x - self.pos[j]).square().sum(1).sqrt()[:, None]
            gs.append(torch.stack([(dr ** o / r * w).sum(1) / fact[o] for o in range(ORDER + 1)], 1))
            f = [-torch.einsum("mpc,mp->mc", vec, w / r ** 3)]
            for o in range(1, ORDER + 1):
                f.append(torch.einsum("mpc,mp->mc", vec, w * (-dr ** o / (r ** 3 * fact[o])
                                                              + dr ** (o - 1) / (r ** 2 * fact[o - 1]))))
            fs.append(torch.stack(f, 2))
        return torch.cat(gs), torch.cat(fs)

    def block(self, rows, cols, k):
        """G and F between contiguous face ranges; k None: F in the static limit."""
        x, y = self.pos[rows], self.pos[cols]
        vec = x[:, None, :] - y[None, :, :]
        same = rows == cols
        eye = torch.eye(x.shape[0], dtype=torch.float64, device=self.dev) if same else 0.0
        d = (vec.square().sum(2) + eye).sqrt()
        nd = torch.einsum("ijc,ic->ij", vec, self.nvec[rows])
        A = self.area[cols][None, :]
        sel = ((self.ri >= rows.start) & (self.ri < rows.stop) & (self.rj >= cols.start) & (self.rj < cols.stop))
        i, j = self.ri[sel] - rows.start, self.rj[sel] - cols.start
        ii = torch.arange(x.shape[0], device=self.dev)
        if k is None:
            F = -nd / d ** 3 * A
            F = F.index_put((i, j), self.fpn[sel][:, 0])
            return None, F.index_put((ii, ii), self.f0n[rows][:, 0])
        pw = torch.stack([(1j * k) ** o for o in range(ORDER + 1)])
        G = (A / d).to(torch.complex128)
        F = nd * (1j * k - 1 / d) / d ** 2 * A
        G = G.index_put((i, j), self.gp[sel].to(torch.complex128) @ pw)
        F = F.index_put((i, j), self.fpn[sel].to(torch.complex128) @ pw)
        ph = torch.exp(1j * k * (d - eye))
        G, F = G * ph, F * ph
        if same:
            G = G.index_put((ii, ii), self.g0[rows].to(torch.complex128) @ pw)
            F = F.index_put((ii, ii), self.f0n[rows].to(torch.complex128) @ pw)
        return G, F

    def matrices(self, k):
        """G1, H1, G2, H2 for the media's wavenumbers k."""
        n, dev = self.n, self.dev
        G1, H1 = (torch.zeros(n, n, dtype=torch.complex128, device=dev) for _ in range(2))
        o = 0
        ident = TWO_PI * torch.eye(n, dtype=torch.float64, device=dev)
        for q, s in enumerate(self.sizes):
            sl = slice(o, o + s)
            g, f = self.block(sl, sl, k[self.inout[q][0] - 1])
            if len(self.sizes) == 1:
                G1, H1 = g, f
            else:
                G1[sl, sl], H1[sl, sl] = g, f
            o += s
        full = slice(0, n)
        G2, H2 = self.block(full, full, k[0])
        return G1, H1 + ident, G2, H2 - ident

    def setup(self, enei, eps):
        self.k0 = TWO_PI / enei
        as_t = lambda e: e if torch.is_tensor(e) else torch.tensor(e, dtype=torch.complex128, device=self.dev)
        self.eps = [as_t(e) for e in eps]
        k = [self.k0 * e.sqrt() for e in self.eps]
        self.k = k
        G1, H1, G2, H2 = self.matrices(k)
        lu = torch.linalg.lu_factor
        self.lu1, self.lu2 = lu(G1), lu(G2)
        S1 = torch.linalg.lu_solve(*self.lu1, H1, left=False)
        S2 = torch.linalg.lu_solve(*self.lu2, H2, left=False)
        self.e1 = torch.stack(self.eps)[self.med[:, 0] - 1]
        self.e2 = torch.stack(self.eps)[self.med[:, 1] - 1]
        self.S1 = S1
        n = self.n
        self.Di = torch.linalg.solve(S1 - S2, torch.eye(n, dtype=torch.complex128, device=self.dev))
        L = self.e1 - self.e2
        self.L = L
        nn = (self.nvec @ self.nvec.T).to(torch.complex128)
        S = S1 * self.e1[None, :] - S2 * self.e2[None, :] + self.k0 ** 2 * (L[:, None] * self.Di * nn) * L[None, :]
        self.luS = lu(S)

    def solve(self, phi, a, alpha, De):
        """sig1, sig2 [n, P], h1, h2 [n, 3, P]."""
        n, k0 = self.n, self.k0
        P = phi.shape[1]
        nv = self.nvec.to(torch.complex128)
        mm = lambda A, x: (A @ x.reshape(n, -1)).reshape(x.shape)
        sv = lambda f, x: torch.linalg.lu_solve(*f, x.reshape(n, -1)).reshape(x.shape)
        inner = lambda x: torch.einsum("nc,ncp->np", nv, x)
        outer = lambda x: nv[:, :, None] * x[:, None, :]
        c1 = lambda e, x: e.reshape((n,) + (1,) * (x.dim() - 1)) * x
        alpha = alpha - mm(self.S1, a) + 1j * k0 * outer(c1(self.e1, phi))
        De = De - mm(self.S1, c1(self.e1, phi)) + 1j * k0 * inner(c1(self.e1, a))
        s2 = sv(self.luS, De + 1j * k0 * inner(c1(self.L, mm(self.Di, alpha))))
        h2 = mm(self.Di, 1j * k0 * outer(c1(self.L, s2)) + alpha)
        return sv(self.lu1, s2 + phi), sv(self.lu2, s2), sv(self.lu1, h2 + a), sv(self.lu2, h2)

    def plane_wave(self, pol, dirs):
        k, k0 = self.k[0], self.k0
        pol, dirs = self.T(pol), self.T(dirs)
        ph = torch.exp(1j * k * (self.pos @ dirs.T)) / (1j * k0)               # [n, P]
        a = ph[:, None, :] * pol.T[None, :, :]
        ap = a * (1j * k * (self.nvec @ dirs.T))[:, None, :]
        sgn = ((self.med[:, 1] == 1).to(torch.float64) - (self.med[:, 0] == 1).to(torch.float64))[:, None, None]
        m2 = (self.med[:, 1] == 1)[:, None]
        m1 = (self.med[:, 0] == 1)[:, None]
        nv = self.nvec.to(torch.complex128)
        inn = torch.einsum("nc,ncp->np", nv, a)
        De = -1j * k0 * (self.e2[:, None] * m2 - self.e1[:, None] * m1) * inn
        return torch.zeros_like(ph), a * sgn, ap * sgn, De

    def far(self, dirs, s):
        k, k0 = self.k[0], self.k0
        ph = torch.exp(-1j * k * (dirs @ self.pos.T)) * self.area[None, :]
        e = h = 0
        for side, (sg, hh) in enumerate(((s[0], s[2]), (s[1], s[3]))):
            w = ph * (self.med[:, side] == 1)[None, :]
            Ph = torch.einsum("dn,ncp->dcp", w, hh)
            e = e + 1j * k0 * Ph - 1j * k * dirs[:, :, None] * (w @ sg)[:, None, :]
            h = h + 1j * k * torch.linalg.cross(dirs[:, :, None].to(Ph.dtype).expand(Ph.shape), Ph, dim=1)
        return e, h

    def sphere(self):
        v, f = shapes.trisphere(256, 2.0)
        c = [self.T(v[f[:, q]]) for q in range(3)]
        N = torch.linalg.cross(c[0] - c[1], c[2] - c[1])
        return _unit(N), 0.5 * N.square().sum(1).sqrt()

    def power(self, e, h, nvec, area):
        flux = 0.5 * torch.einsum("dc,dcp->dp", nvec, torch.linalg.cross(e, h.conj(), dim=1).real)
        return area @ flux

    def cross_sections(self, s, pol, dirs):
        pol, dirs = self.T(pol), self.T(dirs)
        e, _ = self.far(dirs, s)
        amp = torch.einsum("pc,pcp->p", pol.to(e.dtype), e)
        ext = (4 * math.pi / self.k[0] * amp.imag).real
        nv, ar = self.sphere()
        sca = (self.power(*self.far(nv, s), nv, ar) / (0.5 * self.eps[0].sqrt())).real
        return ext, sca

    def media_of(self, pts):
        out = []
        for q in pts.split(2048):
            j = torch.cdist(q, self.pos, compute_mode="donot_use_mm_for_euclid_dist").argmin(1)
            front = ((q - self.pos[j]) * self.nvec[j]).sum(1) >= 0
            out.append(torch.where(front, self.med[j, 1], self.med[j, 0]))
        return torch.cat(out)

    def fields(self, pts, med, s):
        """E and H [m, 3, P] at points in media med."""
        es, hs = [], []
        step = max(64, 40_000_000 // self.n // 4)
        for q, mq in zip(pts.split(step), med.split(step)):
            vec = q[:, None, :] - self.pos[None, :, :]
            d = vec.square().sum(2).sqrt().clamp_min(2.2e-16)
            near = (d - self.rad[None, :]) / self.rad[None, :] < CUTOFF
            pi, pj = near.nonzero(as_tuple=True)
            g, f = self.pair_coefficients(q[pi], pj)
            k = torch.stack(self.k)[mq - 1]
            pw = torch.stack([(1j * k[pi]) ** o for o in range(ORDER + 1)], 1)
            G = (self.area[None, :] / d).to(torch.complex128)
            G = G.index_put((pi, pj), (g * pw).sum(1))
            ph = torch.exp(1j * k[:, None] * d)
            ff = (1j * k[:, None] - 1 / d) / d ** 2 * self.area[None, :]
            Gp = [(ff * vec[:, :, c]).index_put((pi, pj), (f[:, c] * pw).sum(1)) * ph for c in range(3)]
            G = G * ph
            e = h = 0
            for side, (sg, hh) in enumerate(((s[0], s[2]), (s[1], s[3]))):
                w = (self.med[None, :, side] == mq[:, None]).to(torch.float64)
                gw = [x * w for x in Gp]
                e = e + 1j * self.k0 * torch.einsum("ij,jcp->icp", G * w, hh) - torch.stack([x @ sg for x in gw], 1)
                h = h + torch.stack([gw[1] @ hh[:, 2] - gw[2] @ hh[:, 1], gw[2] @ hh[:, 0] - gw[0] @ hh[:, 2],
                                     gw[0] @ hh[:, 1] - gw[1] @ hh[:, 0]], 1)
            es.append(e)
            hs.append(h)
        return torch.cat(es), torch.cat(hs)

    def dipole_potentials(self, pos, med):
        """phi, a, alpha, De of unit dipoles along x, y, z at each position."""
        n, k0 = self.n, self.k0
        nv = self.nvec
        cols = []
        for x, mm in zip(pos, med.tolist()):
            eps = self.eps[mm - 1]
            k = k0 * eps.sqrt()
            v = self.pos - x[None, :]
            r = v.square().sum(1).sqrt()
            u = v / r[:, None]
            G = torch.exp(1j * k * r) / r
            Fd = (1j * k - 1 / r) * G
            en = (nv * u).sum(1)
            for q in range(3):
                dp = torch.zeros(3, dtype=torch.float64, device=self.dev)
                dp[q] = 1.0
                ep, nd = u @ dp, nv @ dp
                phi = -ep * Fd / eps
                phip = ((nd - 3 * en * ep) / r ** 2 * (1 - 1j * k * r) * G + k ** 2 * ep * en * G) / eps
                a = -1j * k0 * dp[None, :] * G[:, None]
                ap = -1j * k0 * dp[None, :] * (en * Fd)[:, None]
                tot = [0, 0, 0, 0]
                for side, sg, e in ((1, 1.0, self.e2), (0, -1.0, self.e1)):
                    w = sg * (self.med[:, side] == mm).to(torch.float64)
                    tot[0] = tot[0] + w * phi
                    tot[1] = tot[1] + w[:, None] * a
                    tot[2] = tot[2] + w[:, None] * (ap - 1j * k0 * nv * (e * phi)[:, None])
                    tot[3] = tot[3] + w * e * (phip - 1j * k0 * (nv * a).sum(1))
                cols.append(tot)
        return tuple(torch.stack([c[q] for c in cols], -1) for q in range(4))


def _np(x):
    return x.detach().cpu().numpy()


def _exact_sweep(case, seed):
    p = _Problem(case, seed)
    ref = _Reference(p.nodes if p.curved else p.meshes, p.inout, curved=p.curved)
    ext, sca = [], []
    for w in p.enei:
        ref.setup(float(w), p.eps(w))
        s = ref.solve(*ref.plane_wave(p.pol, p.dir))
        e, c = ref.cross_sections(s, p.pol, p.dir)
        ext.append(_np(e))
        sca.append(_np(c))
    return {"ext": np.array(ext), "sca": np.array(sca)}


def exact(case, seed):
    kind = case["kind"]
    with torch.set_grad_enabled(kind in ("gradient", "shape")):
        if kind == "batch":
            cs = _batch_cases(case)
            if sum(c["nw"] * (_faces(c) / 1000.0) ** 3 for c in cs) > 450:
                return None
            return [_exact_sweep(c, 10 * int(seed) + i) for i, c in enumerate(cs)]
        n = _faces(case)
        if case.get("nw", 1) * (n / 1000.0) ** 3 > 450 or n > 6500:
            return None
        if kind == "sweep":
            return _exact_sweep(case, seed)
        p = _Problem(case, seed)
        enei = float(p.enei[0])
        eps = p.eps(enei)
        if kind in ("gradient", "shape"):
            dev = _dev()
            v = torch.tensor(p.meshes[0][0], dtype=torch.float64, device=dev, requires_grad=True)
            er = torch.tensor([eps[1].real, eps[1].imag], dtype=torch.float64, device=dev, requires_grad=True)
            ref = _Reference(p.meshes, p.inout, verts=v)
            ref.setup(enei, [eps[0], torch.complex(er[0], er[1])])
            s = ref.solve(*ref.plane_wave(p.pol, p.dir))
            ext, _ = ref.cross_sections(s, p.pol, p.dir)
            ext[0].backward()
            val = float(ext[0].detach()) if kind == "gradient" else _np(ext[0])
            return {"ext": val, "verts": _np(v.grad), "eps": _np(er.grad)}
        ref = _Reference(p.nodes if p.curved else p.meshes, p.inout, curved=p.curved)
        ref.setup(enei, eps)
        if kind == "decay":
            pos = p.dipoles(case)
            pts = ref.T(pos)
            med = ref.media_of(pts)
            s = ref.solve(*ref.dipole_potentials(pts, med))
            P, npt = 3 * case["npt"], case["npt"]
            nv, ar = ref.sphere()
            e, h = ref.far(nv, s)
            k, e0 = ref.k[0], ref.eps[0]
            for c in range(P):
                if int(med[c // 3]) != 1:
                    continue
                dp = torch.zeros(3, dtype=torch.float64, device=ref.dev)
                dp[c % 3] = 1.0
                g = torch.exp(-1j * k * (nv @ pts[c // 3]))
                hh = torch.linalg.cross(nv, dp[None, :].expand(nv.shape)) * g[:, None]
                e[:, :, c] += k ** 2 * torch.linalg.cross(hh, nv.to(hh.dtype)) / e0
                h[:, :, c] += k ** 2 * hh / e0.sqrt()
            power = ref.power(e, h, nv, ar)
            el, _ = ref.fields(pts, med, s)
            tot, rad = np.zeros((npt, 3)), np.zeros((npt, 3))
            for c in range(P):
                nb = float(ref.eps[int(med[c // 3]) - 1].sqrt().real)
                unit = 0.5 * nb * 4.0 / 3.0 * ref.k0 ** 3
                tot[c // 3, c % 3] = 1 + float(el[c // 3, c % 3, c].imag) / unit
                rad[c // 3, c % 3] = float(power[c]) / (TWO_PI * ref.k0) / unit
            return {"tot": tot, "rad": rad, "sig2": _np(s[1])}
        s = ref.solve(*ref.plane_wave(p.pol, p.dir))
        if kind == "map":
            pts = ref.T(p.points(case))
            e, h = ref.fields(pts, ref.media_of(pts), s)
            return {"e": _np(e), "h": _np(h)}
        ext, sca = ref.cross_sections(s, p.pol, p.dir)
        return {"ext": _np(ext), "sca": _np(sca), "sig1": _np(s[0]), "sig2": _np(s[1]), "h1": _np(s[2]),
                "h2": _np(s[3])}
