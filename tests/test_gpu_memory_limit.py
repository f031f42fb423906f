"""A solve that fits into the device memory on one stream also runs where the second
stream's panels and operand buffers (18 KB per face, 72 MB here) do not fit beside it."""
import gc

import numpy as np
import pytest

import mnpbem_gb300 as m
from mnpbem_gb300 import _lib, shapes

from test_gpu_parity import drude

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,faces", [("mixed", 4000), ("fp64", 3000)])
def test_one_stream_near_the_limit(gpu_lib, prec, faces):
    torch = pytest.importorskip("torch")
    v, f = shapes.fibsphere(faces, 50.0)
    cp = m.comparticle([m.epsconst(1.77), drude()], [m.particle(v, f)], [[2, 1]], 1)
    exc = m.planewave([[1.0, 0, 0]], [[0, 0, 1.0]])

    def solve(profile):
        free0 = torch.cuda.mem_get_info()[0]
        bem = m.bemsolver(cp, m.bemoptions(precision=prec))
        _lib.check(gpu_lib.mnpbem_profile_enable(bem._h, int(profile)))    # profiling keeps one stream
        sig = bem.mldivide(exc(cp, 560.0))
        used = free0 - torch.cuda.mem_get_info()[0]
        del bem
        gc.collect()
        return sig, used

    solve(True)                                # module and context memory
    ref, used = solve(True)
    margin = 24 << 20 if prec == "mixed" else 12 << 20
    fill = torch.empty(torch.cuda.mem_get_info()[0] - used - margin, dtype=torch.uint8, device="cuda")
    try:
        sig, _ = solve(False)
    finally:
        del fill
        torch.cuda.empty_cache()
    assert np.array_equal(sig.sig2, ref.sig2)
