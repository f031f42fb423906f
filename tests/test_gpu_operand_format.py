"""The products of Delta's inverse keep 32-bit operands (TF32) below 12 000 faces unless
the caller sets the width of its steps: with LDU updates of rank 256, which never take
FP16 operands, the FP16 option changes no bit of a solution.  A width of 512 set by the
caller takes FP16 operands as before, so there the bits differ."""
import numpy as np
import pytest

import mnpbem_gb300 as m
from mnpbem_gb300 import autotune, shapes

from test_gpu_parity import drude


def test_tuned_settings_leave_the_operands(monkeypatch):
    for faces, entry in autotune.load().items():
        if int(faces) < 12000:
            assert entry["options"].get("gj_block", 256) == 256, faces


@pytest.mark.gpu
@pytest.mark.parametrize("faces", [1000, 2000, 3600])
def test_no_fp16_in_the_inverse_of_delta(gpu_lib, faces):
    v, f = shapes.fibsphere(faces, 50.0)
    cp = m.comparticle([m.epsconst(1.77), drude()], [m.particle(v, f)], [[2, 1]], 1)
    exc = m.planewave([[1.0, 0, 0]], [[0, 0, 1.0]])

    def solve(f16, gj=None):
        bem = m.bemsolver(cp, m.bemoptions(precision="mixed"))
        bem.set_option("lu_steps", 1)
        bem.set_option("tc_f16", f16)
        if gj:
            bem.set_option("gj_block", gj)
        return bem.mldivide(exc(cp, 560.0))

    a, b = solve(1), solve(0)
    for k in ("sig1", "sig2", "h1", "h2"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
    if faces >= 2000:
        assert not np.array_equal(solve(1, 512).sig2, a.sig2)
