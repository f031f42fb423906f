"""Complex128 GEMM on the tensor cores (mnpbem_gemm_c128 path 1: exact FP16
digit products) at the edges of its tiles (128 rows, 32 complex columns, K up
to 64), against a product in extended precision.

Error measure: max over the entries of |C - ref| / (|A_i| |B_j|) with the
2-norms of the row and the column (the operands are scaled per row and column),
plus |C0| for an accumulated product.  The slices keep 2^-63 of the largest entry and
drop levels below 2^-58 of (row maximum) x (column maximum), so 2^-53 (the one rounding of
the result) bounds the error, 2^-52 with the added C; the CUDA-core FP64 product
(path 0) is allowed its K roundings, and the tensor-core product must not be less
accurate than it.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def run(lib, path, alpha, A, B, beta, C0, ldc=None):
    from mnpbem_gb300 import _lib
    M, K = A.shape
    N = B.shape[1]
    ldc = ldc or N
    C = np.full((M, ldc), 3 - 2j)
    C[:, :N] = C0
    _lib.check(lib.mnpbem_gemm_c128(0, path, M, N, K, alpha, A.ctypes.data, K, B.ctypes.data, N, beta,
                                    C.ctypes.data, ldc))
    assert np.all(C[:, N:] == 3 - 2j)
    return C[:, :N]


def exact(alpha, A, B, beta, C0):
    """Real and imaginary part in extended precision."""
    ld = np.longdouble
    ar, ai, br, bi = (x.astype(ld) for x in (A.real, A.imag, B.real, B.imag))
    re = alpha * (ar @ br - ai @ bi) + beta * C0.real.astype(ld)
    im = alpha * (ar @ bi + ai @ br) + beta * C0.imag.astype(ld)
    return re, im


def error(C, ref, A, B, C0, beta):
    scale = np.linalg.norm(A, axis=1)[:, None] * np.linalg.norm(B, axis=0)[None, :] + beta * np.abs(C0)
    d = np.maximum(np.abs(C.real - ref[0]), np.abs(C.imag - ref[1])).astype(float)
    return float(np.max(d / scale))


def operands(M, N, K, kind, seed):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((M, K)) + 1j * rng.standard_normal((M, K))
    B = rng.standard_normal((K, N)) + 1j * rng.standard_normal((K, N))
    if kind == "decay":            # entries of a Green function block: 1/d and 1/d^2 over three decades
        A *= 10.0 ** rng.uniform(-3, 0, (M, K))
        B *= 10.0 ** rng.uniform(-6, 0, (K, N))
    if kind == "scales":           # rows and columns of very different size, and zero ones
        A *= 10.0 ** rng.uniform(-150, 140, (M, 1))
        B *= 10.0 ** rng.uniform(-140, 120, (1, N))
        A[M // 2] = 0
        B[:, N // 3] = 0
    return np.ascontiguousarray(A), np.ascontiguousarray(B)


@pytest.mark.parametrize("M,N,K,kind", [(16, 16, 16, "normal"), (128, 32, 64, "normal"), (129, 33, 63, "decay"),
                                        (127, 31, 17, "scales"), (300, 200, 64, "decay"), (64, 500, 64, "scales"),
                                        (500, 64, 64, "decay"), (260, 290, 50, "normal")])
def test_gemm_c128(gpu_lib, M, N, K, kind):
    A, B = operands(M, N, K, kind, M + N)
    rng = np.random.default_rng(5)
    C0 = rng.standard_normal((M, N)) + 1j * rng.standard_normal((M, N))
    for alpha, beta, ldc in ((1.0, 0.0, None), (-1.0, 1.0, N + 3)):
        ref = exact(alpha, A, B, beta, C0)
        tc = error(run(gpu_lib, 1, alpha, A, B, beta, C0, ldc), ref, A, B, C0, beta) if kind != "scales" else None
        if kind == "scales":       # zero rows and columns: only where the scale is not zero
            C = run(gpu_lib, 1, alpha, A, B, beta, C0, ldc)
            keep = np.ix_(np.arange(M) != M // 2, np.arange(N) != N // 3)
            ref_k = (ref[0][keep], ref[1][keep])
            rows, cols = keep[0].ravel(), keep[1].ravel()
            tc = error(C[keep], ref_k, A[rows], B[:, cols], C0[keep], beta)
            assert np.all(C[M // 2] == beta * C0[M // 2]) and np.all(C[:, N // 3] == beta * C0[:, N // 3])
        assert tc <= (2 if beta else 1) * U, tc
        if kind != "scales":
            simt = error(run(gpu_lib, 0, alpha, A, B, beta, C0, ldc), ref, A, B, C0, beta)
            assert tc <= simt, (tc, simt)


def test_largest_digits_are_summed_exactly(gpu_lib):
    """Entries whose digits are all at their largest: every slice product and
    partial sum is at its bound, and the result is still exact to one rounding."""
    M, N, K = 128, 64, 64
    x = float((1 << 53) - 1)
    A = np.full((M, K), x + 1j * x)
    B = np.full((K, N), x - 1j * x)
    C0 = np.zeros((M, N), dtype=complex)
    C = run(gpu_lib, 1, 1.0, A, B, 0.0, C0)
    re, im = exact(1.0, A, B, 0.0, C0)
    assert np.array_equal(C.real, re.astype(np.float64)) and np.array_equal(C.imag, im.astype(np.float64))


def test_non_finite_entries_give_nan(gpu_lib):
    A, B = operands(40, 48, 32, "normal", 1)
    A[7, 3], B[5, 11] = np.inf, np.nan
    C = run(gpu_lib, 1, 1.0, A, B, 0.0, np.zeros((40, 48), dtype=complex))
    bad = np.zeros((40, 48), dtype=bool)
    bad[7], bad[:, 11] = True, True
    assert np.array_equal(np.isnan(C), bad)


def test_unsupported_shapes_are_refused(gpu_lib):
    A, B = operands(20, 20, 65, "normal", 2)
    C = np.zeros((20, 20), dtype=complex)
    for K, alpha, beta in ((65, 1.0, 0.0), (8, 1.0, 0.0), (32, 0.5, 0.0), (32, 1.0, 0.5)):
        st = gpu_lib.mnpbem_gemm_c128(0, 1, 20, 20, K, alpha, A.ctypes.data, 65, B.ctypes.data, 20, beta, C.ctypes.data,
                                      20)
        assert st == 7             # MNPBEM_ERR_UNSUPPORTED
