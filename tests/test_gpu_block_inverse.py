"""Diagonal-block inverses of the factorisations (mnpbem_block_inverse).

Complex128 blocks up to 64 (cluster kernel, pivoting), complex64 blocks up to
64 (one CTA, pivoting) and up to 256 (cluster kernel, panels of 16), at the
edges of panels, CTAs and clusters, against numpy's complex128 inverse.

Tolerance: Gauss-Jordan elimination has a forward error of about
c w eps cond(A) relative to max|inv(A)|, with a growth factor near 1 on these
matrices; c = 8 covers the complex arithmetic.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL = [1, 2, 7, 8, 9, 16, 31, 33, 63, 64]


def invert(lib, A, lda=None):
    from mnpbem_gb300 import _lib
    w = A.shape[0]
    lda = lda or w
    buf = np.full((w, lda), 7 + 7j, dtype=A.dtype)
    buf[:, :w] = A
    cond = np.zeros(1)
    prec = _lib.FP64 if A.dtype == np.complex128 else _lib.FP32
    st = lib.mnpbem_block_inverse(0, prec, w, buf.ctypes.data, lda, _lib.dptr(cond))
    assert np.all(buf[:, w:] == 7 + 7j)
    return st, buf[:, :w], cond[0]


def block(w, dtype, seed, shuffled):
    """Diagonally dominant complex block; shuffled: its rows permuted, so that
    the elimination has to pivot."""
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((w, w)) + 1j * rng.standard_normal((w, w))
    A = A * (0.4 / np.sqrt(w)) + np.diag(2.0 + rng.random(w) - 1j * rng.random(w))
    if shuffled:
        A = A[rng.permutation(w)]
    return np.ascontiguousarray(A.astype(dtype))


def check(lib, A, lda=None):
    from mnpbem_gb300 import _lib
    w = A.shape[0]
    st, X, cond = invert(lib, A, lda)
    _lib.check(st)
    ref = np.linalg.inv(A.astype(np.complex128))
    eps = np.finfo(A.real.dtype).eps
    tol = 8 * w * eps * np.linalg.cond(A.astype(np.complex128))
    assert np.abs(X - ref).max() <= tol * np.abs(ref).max()
    assert abs(cond - np.abs(A).max() * np.abs(ref).max()) <= 1e-3 * cond


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("w", SMALL)
def test_pivoted_blocks(gpu_lib, w, dtype):
    check(gpu_lib, block(w, dtype, w, False))
    check(gpu_lib, block(w, dtype, w + 100, True), lda=w + 3)


@pytest.mark.parametrize("w", [65, 80, 127, 128, 145, 255, 256])
def test_wide_blocks(gpu_lib, w):
    check(gpu_lib, block(w, np.complex64, w, False))
    check(gpu_lib, block(w, np.complex64, w + 1, False), lda=w + 6)


@pytest.mark.parametrize("dtype,w", [(np.complex64, 40), (np.complex64, 200), (np.complex128, 40)])
def test_singular_block_is_reported(gpu_lib, dtype, w):
    A = block(w, dtype, 3, False)
    A[:, w // 2] = 0
    assert invert(gpu_lib, A)[0] == 4      # MNPBEM_ERR_SINGULAR
