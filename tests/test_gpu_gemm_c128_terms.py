"""Complex128 products on the tensor cores (mnpbem_gemm_c128 path 1), entry by entry:
the error is bounded by the terms of that entry's own sum, as an FP64 sum's is, also
where the entries of a row or column differ by many powers of two, and where all digits
reach their largest values with one sign.

Bound: an entry kept from the digits has an error of at most 2 K u |c| (u = 2^-53; the
kernel's rule on the operands' rounding and the dropped levels) and one rounding; one
computed again in FP64 at most four products and five additions per part.  So
|C - ref| <= (2 K + 2) u sum_k |a_k| |b_k| per real and imaginary part, and u (2 |C0| +
sum) more for the addition of C0.  Subnormal results add 2^-1074.
"""
import numpy as np
import pytest

from test_gpu_gemm_c128 import exact, run

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def check(lib, A, B, ldc=None):
    M, K = A.shape
    N = B.shape[1]
    rng = np.random.default_rng(M + N + K)
    C0 = (rng.standard_normal((M, N)) + 1j * rng.standard_normal((M, N))) * np.abs(A).max() * np.abs(B).max()
    with np.errstate(under="ignore"):
        terms = np.abs(A) @ np.abs(B)
    for alpha, beta in ((1.0, 0.0), (-1.0, 1.0)):
        C = run(lib, 1, alpha, A, B, beta, C0, ldc)
        re, im = exact(alpha, A, B, beta, C0)
        d = np.maximum(np.abs(C.real - re), np.abs(C.imag - im)).astype(float)
        tol = (2 * K + 2) * U * terms + beta * U * (2 * np.abs(C0) + terms) + 2.0 ** -1074
        assert np.all(d <= tol), float(np.max(d / tol))


def graded(M, N, K, seed, a, b):
    """Random operands with column k of A scaled by 2^a[k] and row k of B by 2^b[k]."""
    rng = np.random.default_rng(seed)
    A = (rng.standard_normal((M, K)) + 1j * rng.standard_normal((M, K))) * np.ldexp(1.0, a)[None, :]
    B = (rng.standard_normal((K, N)) + 1j * rng.standard_normal((K, N))) * np.ldexp(1.0, b)[:, None]
    return np.ascontiguousarray(A), np.ascontiguousarray(B)


@pytest.mark.parametrize("M,N,K", [(16, 16, 16), (31, 17, 33), (128, 16, 64), (129, 47, 63), (260, 100, 64)])
@pytest.mark.parametrize("span", [8, 20, 40, 300])
def test_graded_operands(gpu_lib, M, N, K, span):
    rng = np.random.default_rng(span + K)
    s = rng.integers(0, span, K).astype(int)
    check(gpu_lib, *graded(M, N, K, 1, -s, s))                          # faces of very different size
    check(gpu_lib, *graded(M, N, K, 2, -s, s[::-1]), ldc=N + 5)
    check(gpu_lib, *graded(M, N, K, 3, -s, -rng.permutation(s)))


@pytest.mark.parametrize("K", [16, 50, 64])
def test_large_entries_meet_zeros(gpu_lib, K):
    """Each row's and column's largest entry meets a zero: what is left is 2^-31 of
    (row maximum) x (column maximum)."""
    M, N = 40, 36
    rng = np.random.default_rng(K)
    A = (rng.uniform(0.5, 1, (M, K)) - 1j * rng.uniform(0.5, 1, (M, K))) * 2.0 ** -30 / 3
    B = (rng.uniform(0.5, 1, (K, N)) + 1j * rng.uniform(0.5, 1, (K, N))) / 3
    A[:, 3], B[3] = 0.5, 0.0
    check(gpu_lib, A, B)
    check(gpu_lib, np.ascontiguousarray(B.T), np.ascontiguousarray(A.T))


def test_sparse_blocks(gpu_lib):
    """Entries that share no or one term (coplanar faces, identity columns)."""
    rng = np.random.default_rng(4)
    M, N, K = 200, 64, 64
    A = (rng.standard_normal((M, K)) + 1j * rng.standard_normal((M, K))) * (rng.random((M, K)) < 0.05)
    B = np.eye(K, N) * (1 + 2j) + (rng.random((K, N)) < 0.02) * 2.0 ** -45
    check(gpu_lib, np.ascontiguousarray(A), np.ascontiguousarray(B))


def test_coherent_small_digits(gpu_lib):
    """One entry of 1/2 beside entries near 2^-7 with large low digits of one sign: the
    digit products beyond the kept levels all add up."""
    M, N, K = 128, 32, 64
    low = sum(127 * 256.0 ** -(k + 1) for k in range(1, 7)) + 2.0 ** -7
    A = np.full((M, K), low + 0j)
    B = np.full((K, N), low + 0j)
    A[:, 0], B[0] = 0.5, 0.0
    check(gpu_lib, A, B)
    B[0] = 0.5
    check(gpu_lib, A, B)


def test_digits_at_their_largest(gpu_lib):
    """Entries of digits 64, -128, -128, ...: six of the eight products of level 7 and
    five of level 8 at 2^14, all of one sign in one part, so that the sums pass 2^23."""
    M, N, K = 160, 48, 64
    x = 64.0 * 256.0 ** 7 - 128.0 * sum(256.0 ** k for k in range(1, 7))
    A = np.full((M, K), x + 1j * x)
    for B, part in ((np.full((K, N), x - 1j * x), np.real), (np.full((K, N), -x - 1j * x), np.imag)):
        check(gpu_lib, A, B)
        C = run(gpu_lib, 1, 1.0, A, B, 0.0, np.zeros((M, N), dtype=complex))
        ref = (1 if part is np.real else -1) * 2 * K * np.longdouble(x) ** 2
        assert np.all(np.abs(part(C) - ref) <= 2 * U * np.abs(ref))
