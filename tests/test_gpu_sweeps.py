"""Triangular sweeps of the LDU solves (one launch per direction, several
systems at once) at the edges of their blocks and of their register-tiled
column counts: face counts around 64 (complex128 blocks) and 256 (complex64
blocks), one to four polarisations (P and 4 P columns), one particle and a
dimer whose two G1 blocks and G2 are solved together.

Charges and currents against the FP64 oracle (max |diff| / max |ref|): 1e-9 in
FP64 and 1e-8 in mixed precision, the bounds of the parity tests (the
self-element coefficients carry 1e-11, the refinement stops at 1e-10).
"""
import numpy as np
import pytest

import mnpbem_gb300 as m
from mnpbem_gb300 import shapes

pytestmark = pytest.mark.gpu
POL = np.array([[1.0, 0, 0], [0, 1.0, 0], [0, 0, 1.0], [0, 1.0, 0]])
DIR = np.array([[0, 0, 1.0], [0, 0, 1.0], [1.0, 0, 0], [1.0, 0, 0]])


def problem(faces, dimer):
    if dimer:
        n1 = faces // 2 // 2 * 2
        parts = [shapes.fibsphere(n1, 20.0, (-12.0, 0, 0)), shapes.fibsphere(faces - n1, 20.0, (12.0, 0, 0))]
        inout = [[2, 1], [3, 1]]
    else:
        parts, inout = [shapes.fibsphere(faces, 20.0)], [[2, 1]]
    metal = m.epsfun(lambda w: 10 - 9.065 ** 2 / (w * (w + 0.0708j)), "eV")
    return m.comparticle([m.epsconst(1.77)] + [metal] * len(parts), [m.particle(v, f) for v, f in parts], inout,
                         *range(1, len(parts) + 1))


@pytest.mark.parametrize("faces,npol,dimer", [(60, 1, False), (64, 4, False), (66, 2, False), (254, 3, False),
                                              (256, 1, False), (258, 4, False), (300, 3, True), (530, 2, True),
                                              (770, 1, False)])
def test_charges_match_oracle(gpu_lib, faces, npol, dimer):
    from oracle import mnpbem_ref as R
    cp = problem(faces, dimer)
    t = shapes.tables()
    q = R.QuadFace((t["rule18_x"], t["rule18_y"], t["rule18_w"]))
    ocp = R.ComParticle([R.EpsConst(1.77)] + [R.drude_eps() for _ in cp.p],
                        [R.Particle(p.verts, p.faces, q) for p in cp.p], cp.inout, [True] * len(cp.p))
    vi, fi = shapes.trisphere(256, 2.0)
    pw = R.PlaneWaveRet(POL[:npol], DIR[:npol], R.Particle(vi, fi, q))
    ref = R.BemRet(ocp).solve(pw.potential(ocp, 560.0))
    exc = m.planewave(POL[:npol], DIR[:npol])
    for precision, tol in (("fp64", 1e-9), ("mixed", 1e-8)):
        bem = m.bemsolver(cp, m.bemoptions(precision=precision))
        sig = bem.mldivide(exc(cp, 560.0))
        for k in ("sig1", "sig2", "h1", "h2"):
            err = np.abs(getattr(sig, k) - ref[k]).max() / np.abs(ref[k]).max()
            assert err < tol, (precision, k, err)
