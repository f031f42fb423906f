"""Refined faces of field points with the FP32 pre-test: the fields of given charges
do not change when particle and points move far from the origin, where the FP32
distances lose digits (the slack must then hand more pairs to the FP64 test), and
points on and beyond the cutoffs, inside and at a centroid are finite.

Tolerance: a shift of 2^s rounds coordinates to 2^(s - 52); over distances of at
least 0.5 nm the fields (up to 1 / d^3) change by less than 8 * 2^(s - 52) / 0.5
relative to the largest, times 64 for the sums over the faces."""
import numpy as np
import pytest

import mnpbem_gb300 as m
from mnpbem_gb300 import shapes

from test_gpu_parity import drude

pytestmark = pytest.mark.gpu


def fields(v, f, shift, pts, sig):
    cp = m.comparticle([m.epsconst(1.77), drude()], [m.particle(v + shift, f)], [[2, 1]], 1)
    bem = m.bemsolver(cp, m.bemoptions(precision="fp64"))
    if sig is None:
        sig = bem.mldivide(m.planewave([[1.0, 0, 0]], [[0, 0, 1.0]])(cp, 540.0))
    e, h = m.meshfield(bem, pts + shift, medium=np.ones(len(pts), np.int32))(sig)
    return np.asarray(e), np.asarray(h), sig


@pytest.mark.parametrize("s", [4, 10, 16])
def test_fields_far_from_origin(gpu_lib, s):
    v, f = shapes.trisphere(144, 20.0)
    rng = np.random.default_rng(3)
    u = rng.standard_normal((300, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    pts = np.ldexp(np.round(np.ldexp(u * rng.uniform(10.6, 40.0, 300)[:, None], 20)), -20)
    v = np.ldexp(np.round(np.ldexp(v, 20)), -20)      # exact under the shifts
    e0, h0, sig = fields(v, f, 0.0, pts, None)
    e1, h1, _ = fields(v, f, np.array([1.0, -1.0, 0.5]) * 2.0 ** s, pts, sig)
    tol = 64 * 8 * 2.0 ** (s - 52) / 0.5 + 1e-12
    assert np.all(np.isfinite(e1))
    assert np.max(np.abs(e1 - e0)) < tol * np.max(np.abs(e0))
    assert np.max(np.abs(h1 - h0)) < tol * np.max(np.abs(h0))
