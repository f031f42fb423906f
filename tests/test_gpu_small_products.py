"""Complex64 products of a few 64 x 64 tiles (mnpbem_gemm_c64, path 0, N > 16).

Sizes at the edges of the 16 x 32 tile, of the 64-deep step in k and of the rule
on the number of tiles (76 and 77 tiles of 64 x 64, K of 15 and 16), with a row
pitch of C wider than N and alpha / beta other than 1 / 0.

Tolerance: four partial sums of at most ceil(K / 4) products each and two
additions, so the relative error against the sum of moduli stays below
(2 ceil(K / 4) + 4) 2^-24; for random data (sum of moduli about sqrt(K) times the
largest result, errors of both signs) sqrt(K) (2 ceil(K / 4) + 4)^(1/2) 2^-24.
"""
import pytest

from test_gpu_gemm import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 17, 16), (15, 31, 17), (16, 32, 64), (17, 33, 65), (64, 64, 63),
                                   (28, 28, 256), (256, 28, 255), (28, 256, 129), (100, 100, 15),
                                   (64 * 76, 64, 40), (64 * 76 + 1, 64, 40), (500, 600, 128)])
def test_small_products(gpu_lib, M, N, K):
    tol = K ** 0.5 * (2 * -(-K // 4) + 4) ** 0.5 * 2.0 ** -24 + 4 * 2.0 ** -24
    assert run(gpu_lib, 0, M, N, K, 1.0 + 0j, 0.0, M + N) < tol
    assert run(gpu_lib, 0, M, N, K, 0.5 - 0.25j, 1.0, M + N, ldc=N + 3) < tol
