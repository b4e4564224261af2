"""GPU: the Green tensor's exponential sums from per-layer decays, in every
relation of receiver and transmitter: one layer alone, several within one
background layer (touching and with gaps), one per background layer, and pairs
with whole background layers between them, against the oracle's sums of
exponentials. Both are FP64; the exponents reach about 1e3, so the oracle's
own exponentials carry 1e3 2^-53 = 1e-13 and the bound is 1e-10 as for the
other tensors.
"""
import numpy as np
import pytest

from extreme_gb300.model import CartesianModel, OmegaModel, Section1D
from oracle import green

pytestmark = pytest.mark.gpu

# tops and thicknesses of the anomaly layers in a background with interfaces
# at 400, 900, 1700, 2600 m
LAYERS = {
    "alone": ([450.0], [300.0]),
    "touching": ([900.0, 1000.0, 1150.0], [100.0, 150.0, 550.0]),
    "gaps": ([420.0, 600.0, 850.0], [30.0, 120.0, 50.0]),
    "one each": ([0.0, 400.0, 900.0, 1700.0], [400.0, 500.0, 800.0, 900.0]),
    "far": ([10.0, 380.0, 1800.0, 2300.0, 2600.0], [100.0, 20.0, 300.0, 300.0, 50.0]),
}


@pytest.mark.parametrize("name", sorted(LAYERS))
@pytest.mark.parametrize("freq", [0.01, 10.0])
def test_tensor_matches_oracle(egx_ctx, name, freq):
    depth, thick = (np.array(v) for v in LAYERS[name])
    section = Section1D(0.0, np.array([0.0, 400.0, 500.0, 800.0, 900.0, 2000.0, 0.0]),
                        np.array([0.0, 0.1, 0.001, 0.5, 0.01, 1.0, 0.05]))
    m = CartesianModel(4, 3, 300.0, 450.0, section, depth, thick, np.zeros((4, 3, len(depth))))
    m.sigma[:] = section.sigma[m.background_indices()][None, None, :]
    om = OmegaModel.build(m.validate(), freq)
    want = green.green_tensor(om, 4)
    g = egx_ctx.green_build(m, om.omega, n_hankels=4)
    try:
        got = g.download()
        for c in ("xx", "xy", "yy", "zz", "xz", "yz"):
            a, b = np.ravel(got[c]), np.ravel(want[c])
            assert np.linalg.norm(a - b) <= 1e-10 * np.linalg.norm(b), c
    finally:
        g.free()
