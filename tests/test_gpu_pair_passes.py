"""FP64 pair passes at the edges of their register-tiled sizes, against the
oracle: the adjoint near and self passes for expansion orders in both of their
instances (up to 5, up to 8), on triangles and quadrilaterals, and the fields
at points for one to four polarisations and point counts around the eight
points of a block.  Tolerances as in the tests of these paths: gradients 1e-8
(max |diff| / max |ref|), fields 1e-10.
"""
import numpy as np
import pytest

import mnpbem_gb300 as m
from mnpbem_gb300 import shapes

pytestmark = pytest.mark.gpu
EPS_IN = complex(-8.5, 0.9)
POL = np.array([[1.0, 0, 0], [0, 1.0, 0], [0, 0, 1.0], [0, 1.0, 0]])
DIR = np.array([[0, 0, 1.0], [0, 0, 1.0], [1.0, 0, 0], [1.0, 0, 0]])


def quadface():
    from oracle import mnpbem_ref as R
    t = shapes.tables()
    return R, R.QuadFace((t["rule18_x"], t["rule18_y"], t["rule18_w"]))


@pytest.mark.parametrize("order,triangles", [(5, False), (1, True), (3, False), (6, True), (8, False)])
def test_gradient_orders(gpu_lib, order, triangles):
    from oracle import adjoint_ref as A
    R, q = quadface()
    v, f = shapes.trirod(6.0, 16.0, (9, 4, 5), triangles=triangles)
    vi, fi = shapes.trisphere(256, 2.0)
    pol, dirv = [0, 0, 1.0], [1.0, 0, 0]
    J0, gv0, ge0, _ = A.cross_section_gradient(v, f, q, 1.77, EPS_IN, 520.0, pol, dirv, "ext", R.Particle(vi, fi, q),
                                               order)
    cp = m.comparticle([m.epsconst(1.77), m.epsconst(EPS_IN)], [m.particle(v, f)], [[2, 1]], 1)
    bem = m.bemsolver(cp, m.bemoptions(precision="fp64", order=order))
    val, gv, ge = bem.cross_section_gradient(m.planewave([pol], [dirv]), 520.0, 0, "ext")
    assert abs(val - J0) / abs(J0) < 1e-10
    assert np.max(np.abs(gv - gv0)) / np.max(np.abs(gv0)) < 1e-8
    assert abs(ge - ge0) / abs(ge0) < 1e-8


@pytest.mark.parametrize("npts,npol", [(1, 1), (7, 2), (8, 3), (9, 4), (33, 1)])
def test_point_fields_sizes(gpu_lib, npts, npol):
    R, q = quadface()
    p = m.trisphere(60, 20.0)
    metal = m.epsfun(lambda w: 10 - 9.065 ** 2 / (w * (w + 0.0708j)), "eV")
    cp = m.comparticle([m.epsconst(1.77), metal], [p], [[2, 1]], 1)
    bem = m.bemsolver(cp, m.bemoptions(precision="fp64"))
    sig = bem.mldivide(m.planewave(POL[:npol], DIR[:npol])(cp, 540.0))
    rng = np.random.default_rng(npts)
    u = rng.standard_normal((npts, 3))
    pts = u / np.linalg.norm(u, axis=1)[:, None] * rng.uniform(3.0, 40.0, npts)[:, None]
    emesh = m.meshfield(bem, pts)
    e, h = emesh(sig)
    ocp = R.ComParticle([R.EpsConst(1.77), R.drude_eps()], [R.Particle(p.verts, p.faces, q)], [[2, 1]], [True])
    eo, ho = R.point_fields(ocp, pts, emesh.medium, 540.0, sig.sig1, sig.sig2, sig.h1, sig.h2)
    assert np.abs(e - eo).max() < 1e-10 * np.abs(eo).max()
    assert np.abs(h - ho).max() < 1e-10 * np.abs(ho).max()
