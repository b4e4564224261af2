"""GPU: the double-FP32 contraction (Dot2 on float pairs) at the layer counts
that take it, 49 to 53, and the first that does not, against the oracle's
operator and the complex128 kernel.

Tolerance: as for the residual apply elsewhere, 1e-12 per vector (47 bits of
each operand and sum, 2^-47 = 7e-15, up to 160 complex terms)."""
import numpy as np
import pytest

from extreme_gb300 import egx
from extreme_gb300.model import OmegaModel, freq_to_omega, random_model
from oracle import operator as op

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(np.ravel(b))


@pytest.mark.parametrize("nz,nrhs", [(49, 1), (49, 10), (50, 2), (51, 3), (53, 1), (53, 9), (53, 10), (54, 1)])
def test_residual_apply_beyond_the_digit_products(egx_ctx, nz, nrhs):
    m = random_model(5, 4, nz, seed=nz, n_boxes=0)
    m.sigma = m.sigma * 10.0 ** np.random.default_rng(nz).uniform(-1, 1, m.sigma.shape)
    f = m.frequencies[1]
    om = OmegaModel.build(m, f)
    g = egx_ctx.green_build(m, freq_to_omega(f), 10)
    try:
        G = g.download()
        egx_ctx.op_prepare(g, om.zeta, om.zeta0, m.layer_thickness, op.OP_A)
        rng = np.random.default_rng(nz + nrhs)
        n = m.nx * m.ny * 3 * nz
        xs = rng.standard_normal((nrhs, n)) + 1j * rng.standard_normal((nrhs, n))
        xs *= 10.0 ** rng.uniform(-8, 2, (nrhs, n))
        y = egx_ctx.op_apply_ds(xs.reshape(-1), nrhs=nrhs).reshape(nrhs, n)
        y64 = egx_ctx.op_apply(xs.reshape(-1), nrhs=nrhs).reshape(nrhs, n)
        takes = nz <= 53 and 4 * nrhs * 3 * nz * 16 <= 96 * 1024
        assert np.array_equal(y, y64) != takes  # another kernel's roundings, where it is taken
        for i in range(nrhs):
            want = op.apply(G, om, xs[i], op.OP_A)
            assert rel(y[i], want) < 1e-12 and rel(y64[i], want) < 4e-14, i
    finally:
        g.free()
