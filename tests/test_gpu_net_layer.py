"""GPU: the passes of the learned network over whole activations at the sizes
where their tiles end (depths of 1, 16 and 32 and one more or less, channels
of one and two 32-column chunks, lines that do not fill 16 cells, channels
without 16-byte rows) against the FP64 oracle.

Tolerance: BF16 operands (2^-9 each), two per product and about seven
products in a chain per layer, with random signs: 2^-9 sqrt(2 x 7 x 2) = 1e-2
of a block's norm for two layers; twice that for gradients that cancel. A row
or column left out at the end of a tile is an error of 1 / sqrt(33) or more.
"""
import numpy as np
import pytest

from extreme_gb300 import egx
from oracle import spectral_net as sn

pytestmark = pytest.mark.gpu
TOL = 2e-2


@pytest.mark.parametrize("nx,ny,nz,W,L,B", [(17, 16, 1, 12, 2, 1), (16, 33, 16, 8, 2, 2), (9, 18, 17, 36, 2, 1),
                                            (20, 7, 32, 32, 2, 2), (18, 31, 33, 32, 1, 1), (7, 16, 31, 64, 2, 1),
                                            (11, 10, 3, 10, 2, 2)])
def test_loss_gradient_and_apply_match_oracle(egx_ctx, nx, ny, nz, W, L, B):
    net = egx.SpectralNet(egx_ctx, nx, ny, nz, width=W, layers=L, seed=nx)
    try:
        rng = np.random.default_rng(nx * nz)
        flat = net.params()
        lay, _ = sn.layout(nz, W, L)
        for name in ("Q", "bQ", "bP") + tuple("b%d" % l for l in range(L)):
            off, shape = lay[name]
            flat[off:off + int(np.prod(shape))] = 0.2 * rng.standard_normal(int(np.prod(shape)))
        net.params(flat)
        n = nx * ny * 3 * nz
        v = (rng.standard_normal((B, n)) + 1j * rng.standard_normal((B, n))).astype(np.complex64)
        t = (0.3 * (rng.standard_normal((B, n)) + 1j * rng.standard_normal((B, n)))).astype(np.complex64)
        logsig = rng.uniform(-3, 1, (nx, ny, nz)).astype(np.float32)
        net.set_model(logsig)
        loss, g = net.loss_grad(v, t, want_grad=True)
        args = (logsig.astype(np.float64), nx, ny, nz, W, L)
        ref_loss, ref_g = sn.loss_grad(flat.astype(np.float64), v.astype(complex), t.astype(complex), *args)
        assert abs(loss - ref_loss) <= TOL * ref_loss
        for name, (off, shape) in lay.items():
            a, b = (x[off:off + int(np.prod(shape))].astype(np.float64) for x in (g, ref_g))
            assert np.linalg.norm(a - b) <= TOL * np.linalg.norm(b), name
        z, ref = net.apply(v), sn.apply(flat.astype(np.float64), v.astype(complex), *args)
        assert np.linalg.norm(z - ref) <= TOL * np.linalg.norm(ref - v)
    finally:
        net.free()
