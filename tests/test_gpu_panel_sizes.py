"""Mixed-precision solves whose last panel is one column, two, odd or nearly full
(16-byte and single-entry panel copies, remainders of the 64- and 256-wide blocks),
on open pieces of a sphere, against the FP64 solve: 1e-8 (max |diff| / max |ref|),
the refinement's tolerance of 1e-10 times the condition of the system."""
import numpy as np
import pytest

import mnpbem_gb300 as m
from mnpbem_gb300 import shapes

from test_gpu_parity import drude

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [63, 65, 255, 257, 258, 301, 511, 513])
def test_last_panel(gpu_lib, n):
    v, f = shapes.trisphere(400, 20.0)
    cp = m.comparticle([m.epsconst(1.77), drude()], [m.particle(v, f[:n])], [[2, 1]])
    exc = m.planewave([[1.0, 0, 0]], [[0, 0, 1.0]])
    r = [m.bemsolver(cp, m.bemoptions(precision=p)).spectrum(exc, [540.0], fields=True) for p in ("mixed", "fp64")]
    for k in ("sig1", "sig2", "h1", "h2"):
        assert np.max(np.abs(r[0][k] - r[1][k])) < 1e-8 * np.max(np.abs(r[1][k])), k
