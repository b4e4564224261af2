"""GPU: the Krylov vector sums at the edges of their tiles (a partial chunk of
16 columns, one thread, one block, more rows than one round of 1024 blocks)
against extended-precision sums. Tolerance: a thread's FP64 chain has n /
262,144 rounded terms of four products, the trees above it 8 + 8 + 4 levels:
(4 n / 262,144 + 20) 2^-53 of the sum of moduli, times two for the products.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ncols", [(1, 1), (255, 16), (256, 17), (257, 8), (5000, 64), (262144, 3), (600001, 9)])
def test_dot_products(egx_ctx, n, ncols):
    rng = np.random.default_rng(n)
    V = rng.standard_normal((ncols, n)) + 1j * rng.standard_normal((ncols, n))
    w = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    tol = 2 * (4 * max(1, n // 262144) + 20) * 2.0 ** -53
    for _ in range(2):  # the scratch is ready for the next launch
        got = egx_ctx.dot_products(V.T, w)
        for k in range(ncols):
            want = np.sum(np.conj(V[k]).astype(np.clongdouble) * w)
            assert abs(got[k] - want) <= tol * np.sum(np.abs(V[k]) * np.abs(w)), k
