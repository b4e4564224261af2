"""GPU: the complex128 contraction by digit products (sizes where its tiles
end: one layer, odd layers, full and partial 16-row tiles, the largest that
it takes and the first that it does not) against the oracle's operator.

Tolerance: both sides round at 2^-53; the oracle's sums have 6 nz <= 300
terms and its transforms a few stages, so their difference stays well below
(300 + 40) 2^-53 = 4e-14 of the result's norm.
"""
import numpy as np
import pytest

from extreme_gb300 import egx
from extreme_gb300.model import OmegaModel, freq_to_omega, random_model
from oracle import operator as op

pytestmark = pytest.mark.gpu
TOL = 4e-14


def rel(a, b):
    return np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(np.ravel(b))


def _model(nz, seed):
    m = random_model(6, 5, nz, seed=seed, n_boxes=0)
    m.sigma = m.sigma * 10.0 ** np.random.default_rng(seed).uniform(-1, 1, m.sigma.shape)
    return m


def _layer_scaled(G, nz, s):
    """The tensor with entry (rc, tr) of every component times s[rc] s[tr]."""
    tr, rc = np.meshgrid(np.arange(nz), np.arange(nz), indexing="ij")
    up = rc <= tr
    w = s[:, None] * s[None, :]
    return {c: v * (w.reshape(-1) if c in ("xz", "yz") else w[rc[up], tr[up]]) for c, v in G.items()}


@pytest.mark.parametrize("nz,nrhs", [(1, 1), (2, 3), (5, 2), (7, 1), (8, 2), (16, 1), (17, 2), (32, 1), (33, 2),
                                     (47, 1), (48, 2), (49, 1)])
@pytest.mark.parametrize("decades", [0, 6])
def test_apply_by_digits_matches_oracle(egx_ctx, nz, nrhs, decades):
    m = _model(nz, nz)
    f = m.frequencies[1]
    om = OmegaModel.build(m, f)
    g = egx_ctx.green_build(m, freq_to_omega(f), 10)
    G = g.download()
    g.free()
    rng = np.random.default_rng(nz)
    G = _layer_scaled(G, nz, 10.0 ** rng.uniform(-decades / 2, decades / 2, nz))
    g = egx_ctx.green_upload(G, m.nx, m.ny, nz)
    try:
        egx_ctx.op_prepare(g, om.zeta, om.zeta0, m.layer_thickness, op.OP_A)
        n = m.nx * m.ny * 3 * nz
        xs = rng.standard_normal((nrhs, n)) + 1j * rng.standard_normal((nrhs, n))
        xs *= 10.0 ** rng.uniform(-3, 3, (nrhs, 1))
        y = egx_ctx.op_apply(xs.reshape(-1), nrhs=nrhs).reshape(nrhs, n)
        for i in range(nrhs):
            assert rel(y[i], op.apply(G, om, xs[i], op.OP_A)) < TOL, i
    finally:
        g.free()


def test_zero_and_nonfinite_vectors(egx_ctx):
    """A zero vector gives exact zeros; a NaN or an infinity anywhere in a
    vector leaves nothing finite in the components that it reaches, and the
    other right-hand side untouched."""
    nz = 9
    m = _model(nz, 2)
    f = m.frequencies[1]
    om = OmegaModel.build(m, f)
    g = egx_ctx.green_build(m, freq_to_omega(f), 10)
    try:
        egx_ctx.op_prepare(g, om.zeta, om.zeta0, m.layer_thickness, op.OP_A)
        n = m.nx * m.ny * 3 * nz
        rng = np.random.default_rng(0)
        x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        want = egx_ctx.op_apply(x)
        y = egx_ctx.op_apply(np.concatenate([np.zeros(n, complex), x]), nrhs=2).reshape(2, n)
        assert not y[0].any() and np.array_equal(y[1], want)
        for bad in (np.nan, np.inf, 1j * np.inf):
            xb = x.copy()
            xb[n // 2] = bad
            y = egx_ctx.op_apply(np.concatenate([x, xb]), nrhs=2).reshape(2, n)
            assert np.array_equal(y[0], want) and not np.isfinite(y[1]).any()
    finally:
        g.free()


# complex64: inputs and results round at 2^-24, the two transforms of 12 and 10
# points at 2^-24 per stage (16 stages in all); the products are exact to
# 2^-29 of the block's largest: (2 + 16) 2^-24 = 1.1e-6, doubled for the
# stages' own constants.
TOL_C64 = 2.2e-6


@pytest.mark.parametrize("nz,nrhs", [(1, 2), (2, 1), (5, 3), (8, 2), (17, 1), (22, 2), (33, 1), (35, 4), (37, 2),
                                     (39, 1), (47, 2), (49, 1)])
@pytest.mark.parametrize("decades", [0, 6])
def test_complex64_apply_by_digits_matches_oracle(egx_ctx, nz, nrhs, decades):
    """Packed layouts, one and two right-hand sides per pass with a remainder."""
    m = _model(nz, nz)
    f = m.frequencies[1]
    om = OmegaModel.build(m, f)
    g = egx_ctx.green_build(m, freq_to_omega(f), 10)
    G = g.download()
    g.free()
    rng = np.random.default_rng(nz)
    G = _layer_scaled(G, nz, 10.0 ** rng.uniform(-decades / 2, decades / 2, nz))
    g = egx_ctx.green_upload(G, m.nx, m.ny, nz, precision=egx.PREC_MIXED)
    try:
        egx_ctx.op_prepare(g, om.zeta, om.zeta0, m.layer_thickness, op.OP_A)
        n = m.nx * m.ny * 3 * nz
        xs = rng.standard_normal((nrhs, n)) + 1j * rng.standard_normal((nrhs, n))
        xs = (xs * 10.0 ** rng.uniform(-3, 3, (nrhs, 1))).astype(np.complex64)
        y = egx_ctx.op_apply_c64(xs.reshape(-1), nrhs=nrhs).reshape(nrhs, n)
        for i in range(nrhs):
            assert rel(y[i], op.apply(G, om, xs[i].astype(complex), op.OP_A)) < TOL_C64, i
    finally:
        g.free()
