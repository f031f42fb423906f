"""G1's factorisation on a second stream beside G2's: the same bits as in one
stream (profiling, which times every phase by itself, keeps one stream), for one
and two diagonal blocks of G1, both precisions, direct and captured runs."""
import numpy as np
import pytest

import mnpbem_gb300 as m
from mnpbem_gb300 import _lib, shapes

from test_gpu_parity import drude

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("two", [False, True])
def test_bits_of_one_stream(gpu_lib, prec, two):
    v, f = shapes.trisphere(256, 20.0)
    parts = [m.particle(v, f)]
    if two:
        parts.append(m.particle(v + np.array([25.0, 0, 0]), f))
    cp = m.comparticle([m.epsconst(1.77), drude()], parts, [[2, 1]] * len(parts), *range(1, len(parts) + 1))
    bem = m.bemsolver(cp, m.bemoptions(precision=prec))
    exc = m.planewave([[1.0, 0, 0]], [[0, 0, 1.0]])
    enei = [520.0, 560.0, 610.0]
    runs = [bem.spectrum(exc, enei, fields=True) for _ in range(2)]
    _lib.check(gpu_lib.mnpbem_profile_enable(bem._h, 1))
    one = bem.spectrum(exc, enei, fields=True)
    _lib.check(gpu_lib.mnpbem_profile_enable(bem._h, 0))
    for r in runs:
        for k in ("sig1", "sig2", "h1", "h2"):
            assert np.array_equal(r[k], one[k]), k
