"""Field points inside a particle and close to face centroids, where the FP32 pre-test
must hand every pair to the FP64 test: against the oracle, to the tolerance of the field
tests (1e-10 of the largest field; the points keep 2 % of an edge from the centroids, at
which the fields of a flat face are singular)."""
import numpy as np
import pytest

import mnpbem_gb300 as m
from mnpbem_gb300 import shapes

from test_gpu_parity import drude, oracle_setup, rel

pytestmark = pytest.mark.gpu


def test_points_inside_and_near_centroids(gpu_lib):
    p = m.trisphere(144, 20.0)
    cp = m.comparticle([m.epsconst(1.77), drude()], [p], [[2, 1]], 1)
    bem = m.bemsolver(cp, m.bemoptions(precision="fp64"))
    sig = bem.mldivide(m.planewave([[1.0, 0, 0]], [[0, 0, 1.0]])(cp, 540.0))
    rng = np.random.default_rng(2)
    u = rng.standard_normal((60, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    inside = u * rng.uniform(0.0, 9.5, 60)[:, None]
    edge = np.sqrt(cp.area)[:, None]
    out = (cp.pos + 0.02 * edge * cp.nvec)[::7]
    inn = (cp.pos - 0.02 * edge * cp.nvec)[::7]
    pts = np.concatenate([inside, inn, out])
    med = np.array([2] * (60 + len(inn)) + [1] * len(out), np.int32)
    e, h = m.meshfield(bem, pts, medium=med)(sig)
    R, ocp, _ = oracle_setup(cp)
    eo, ho = R.point_fields(ocp, pts, med, 540.0, sig.sig1, sig.sig2, sig.h1, sig.h2)
    assert rel(e, eo) < 1e-10 and rel(h, ho) < 1e-10
    assert rel(e[:60], eo[:60]) < 1e-10
