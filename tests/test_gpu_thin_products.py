"""Complex64 products with few columns (mnpbem_gemm_c64, path 0, N <= 16).

One warp takes one to four rows of A by the number of columns and of rows: the
sizes cover every N, the edges of a CTA's rows (8 warps), the row counts at which
the rows per warp change, k ranges below, at and beyond one staged chunk of B with
odd remainders, a row pitch of C wider than N and alpha / beta other than 1 / 0.

Tolerance: each lane of a warp adds at most ceil(K / 32) products in FP32 and five
shuffles add the lanes, so a sum's relative error stays below
(2 ceil(K / 32) + 7) 2^-24 of the sum of moduli; on random data, whose sums of
moduli are about sqrt(K) times the largest result, rounding errors of both signs
leave no more than sqrt(K) (2 ceil(K / 32) + 7)^(1/2) 2^-24 < 3e-5 for K <= 1100.
"""
import numpy as np
import pytest

from test_gpu_gemm import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", range(1, 17))
def test_thin_products(gpu_lib, N):
    for M, K in [(1, 2), (7, 34), (33, 254), (65, 514), (1217, 258), (2433, 300), (4865, 66), (9729, 34),
                 (300, 1100)]:
        tol = K ** 0.5 * (2 * -(-K // 32) + 7) ** 0.5 * 2.0 ** -24 + 4 * 2.0 ** -24
        assert run(gpu_lib, 0, M, N, K, 1.0 + 0j, 0.0, M + N) < tol, (M, K)
        assert run(gpu_lib, 0, M, N, K, 0.5 - 0.25j, 1.0, M + N, ldc=N + 3) < tol, (M, K)
