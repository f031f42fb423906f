"""Sizes and places at which a kernel takes its other branch: thin products of an odd K
in rows of even length (the last k by one lane), two particles of which the first has
an odd number of faces (G1's second block and its vectors unaligned), and G1's chain on
a second stream at sizes whose updates take FP16 operands (K, M, N >= 512).

Tolerances.  Thin products: as in test_gpu_thin_products.py.  Particles in the other
order are the same physical system, so cross sections and charges agree to the
refinement tolerance of 1e-10 (1e-13 times the condition, below 1e3, in FP64) times a
factor of 10 for its two uses.  One and two streams: bits."""
import numpy as np
import pytest

import mnpbem_gb300 as m
from mnpbem_gb300 import _lib, shapes

from test_gpu_parity import drude, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 2, 3, 4, 6, 7, 8, 9, 12, 16])
@pytest.mark.parametrize("M,K", [(5, 3), (33, 33), (70, 257), (1217, 511), (2433, 513), (300, 1101)])
def test_thin_products_of_odd_k(gpu_lib, M, K, N):
    rng = np.random.default_rng(M + K + N)
    lda = K + 1
    c = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    A, B, C0 = c(M, lda), c(K, N), c(M, N)
    A[:, K] = np.nan                       # beyond the row: must not be read into the sum
    tol = K ** 0.5 * (2 * -(-K // 32) + 7) ** 0.5 * 2.0 ** -24 + 4 * 2.0 ** -24
    for alpha, beta in ((1.0 + 0j, 0.0), (0.5 - 0.25j, 1.0)):
        C = C0.copy()
        al, be = np.array([alpha.real, alpha.imag], np.float32), np.array([beta, 0.0], np.float32)
        _lib.check(gpu_lib.mnpbem_gemm_c64(0, 0, M, N, K, al.ctypes.data, A.ctypes.data, lda, B.ctypes.data, N,
                                           be.ctypes.data, C.ctypes.data, N))
        ref = alpha * (A[:, :K].astype(np.complex128) @ B.astype(np.complex128)) + beta * C0
        assert np.max(np.abs(C - ref)) / np.max(np.abs(ref)) < tol


@pytest.mark.parametrize("prec,tol", [("mixed", 1e-9), ("fp64", 1e-9)])
@pytest.mark.parametrize("npol", [1, 2, 3])
def test_odd_first_particle(gpu_lib, prec, tol, npol):
    va, fa = shapes.trirod(8.0, 20.0, (10, 4, 6))
    vb, fb = shapes.trirod(9.0, 24.0, (12, 5, 5))
    a, b = m.particle(va, fa), m.particle(vb + np.array([11.0, 0.5, 1.0]), fb)
    assert a.n % 2 == 1 and a.n > 64
    exc = m.planewave([[1.0, 0, 0], [0, 1.0, 0], [0.6, 0.8, 0]][:npol], [[0, 0, 1.0]] * npol)
    res = []
    for parts in ((a, b), (b, a)):
        cp = m.comparticle([m.epsconst(1.77), drude(), drude()], list(parts), [[2, 1], [3, 1]], 1, 2)
        bem = m.bemsolver(cp, m.bemoptions(precision=prec))
        s = bem.mldivide(exc(cp, 560.0))
        sig = np.asarray(s.sig2)
        n0 = parts[0].n
        res.append((s.ext, s.sca, sig if parts[0] is a else np.concatenate([sig[n0:], sig[:n0]])))
    for x, y in zip(*res):
        assert rel(x, y) < tol


def test_two_streams_with_fp16_updates(gpu_lib):
    v, f = shapes.fibsphere(1200, 40.0)
    cp = m.comparticle([m.epsconst(1.77), drude(), drude()], [m.particle(v, f), m.particle(v + [43.0, 0, 0], f)],
                       [[2, 1], [3, 1]], 1, 2)
    bem = m.bemsolver(cp, m.bemoptions(precision="mixed"))
    exc = m.planewave([[1.0, 0, 0]], [[0, 0, 1.0]])
    enei = [520.0, 560.0, 610.0]
    runs = [bem.spectrum(exc, enei, fields=True) for _ in range(2)]
    _lib.check(gpu_lib.mnpbem_profile_enable(bem._h, 1))
    one = bem.spectrum(exc, enei, fields=True)
    _lib.check(gpu_lib.mnpbem_profile_enable(bem._h, 0))
    for r in runs:
        for k in ("sig1", "sig2", "h1", "h2"):
            assert np.array_equal(r[k], one[k]), k
