"""Two spheres whose sizes differ by up to 300, small enough for blocks of the
factorisation to span both: the FP64 Sigma1 = H1 G1^-1 of initmat against LAPACK on the
library's own matrices, and the mixed solve against the FP64 one.

Tolerance: a row of Sigma1 solves s G1 = h, whose error is at most 16 n u kappa of its
largest entry with kappa the condition of G1 after its columns (the faces' areas) are
scaled to one size, which leaves Sigma1 unchanged.  Mixed: 1e-9 where its refinement
converges (size ratios up to 30)."""
import numpy as np
import pytest

import mnpbem_gb300 as m
from mnpbem_gb300 import shapes

from test_gpu_parity import drude, rel

pytestmark = pytest.mark.gpu


def pair(nv, ratio):
    va, fa = shapes.trisphere(nv, 20.0)
    vb, fb = shapes.trisphere(nv, 20.0 * ratio)
    gap = 10.0 + 10.0 * ratio + 2.0
    return m.comparticle([m.epsconst(1.77), drude()], [m.particle(va, fa), m.particle(vb + [gap, 0, 0], fb)],
                         [[2, 1], [2, 1]], 1, 2)


@pytest.mark.parametrize("nv", [60, 144])
@pytest.mark.parametrize("ratio", [1.0, 10.0, 30.0])
def test_fp64_sigma1(gpu_lib, nv, ratio):
    cp = pair(nv, ratio)
    bem = m.bemsolver(cp, m.bemoptions(precision="fp64"))
    G1, H1 = bem.matrices(550.0, "fp64")[:2]
    size = np.abs(G1).max(0)
    Gs, Hs = G1 / size, H1 / size
    ref = np.linalg.solve(Gs.T, Hs.T).T
    d = np.abs(bem.bem_matrices(550.0, "fp64")["Sigma1"] - ref)
    tol = 16 * cp.n * 2.0 ** -53 * np.linalg.cond(Gs)
    assert np.max(d.max(1) / np.abs(ref).max(1)) < tol
    exc = m.planewave([[1.0, 0, 0]], [[0, 0, 1.0]])
    mixed = m.bemsolver(cp, m.bemoptions(precision="mixed")).spectrum(exc, [550.0, 600.0])
    assert rel(mixed["ext"], bem.spectrum(exc, [550.0, 600.0])["ext"]) < 1e-9
