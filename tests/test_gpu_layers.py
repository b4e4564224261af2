"""GPU: the error of each layer of an apply by itself. A source in one layer,
or one that falls by many decades over the layers, makes responses of very
different size, and the small ones are to be as accurate as the large ones.

Tolerances, of each layer's own 2-norm: complex128 both sides round at 2^-53,
at most 300 terms and 40 operations of the transforms, (300 + 40) 2^-53 =
4e-14; complex64 inputs, the two transforms of 12 and 10 points (16 stages)
and results at 2^-24, doubled for the stages' constants: 2.2e-6; the sub-block
layout of complex64 keeps 22 bits of an operand: 2e-5, as in the other tests of
its kernels.
"""
import numpy as np
import pytest

from extreme_gb300 import egx
from extreme_gb300.model import OmegaModel, freq_to_omega, random_model
from oracle import operator as op

pytestmark = pytest.mark.gpu


def _case(ctx, nz, f, seed):
    m = random_model(6, 5, nz, seed=seed, n_boxes=0)
    m.sigma = m.sigma * 10.0 ** np.random.default_rng(seed).uniform(-1, 1, m.sigma.shape)
    om = OmegaModel.build(m, f)
    g = ctx.green_build(m, freq_to_omega(f), 10)
    G = g.download()
    g.free()
    return m, om, G


def _sources(m, nz, rng, kind):
    x = rng.standard_normal((m.nx, m.ny, 3, nz)) + 1j * rng.standard_normal((m.nx, m.ny, 3, nz))
    if kind == "one layer":
        w = np.zeros(nz)
        w[nz // 4] = 1.0
    else:  # down and up again by twelve decades
        w = 10.0 ** (-12.0 * np.abs(np.sin(np.arange(nz) * 2.0)))
    return (x * w).reshape(-1)


def _layer_errors(y, want, m, nz):
    d = (np.asarray(y, complex) - want).reshape(m.nx * m.ny * 3, nz)
    return np.linalg.norm(d, axis=0) / np.linalg.norm(want.reshape(m.nx * m.ny * 3, nz), axis=0)


@pytest.mark.parametrize("nz,f", [(9, 0.1), (22, 0.1), (24, 10.0), (35, 1.0), (48, 0.1)])
@pytest.mark.parametrize("kind", ["one layer", "falling"])
@pytest.mark.parametrize("entry", ["c128", "ds"])
def test_every_layer_in_complex128(egx_ctx, nz, f, kind, entry):
    m, om, G = _case(egx_ctx, nz, f, nz)
    g = egx_ctx.green_upload(G, m.nx, m.ny, nz)
    try:
        egx_ctx.op_prepare(g, om.zeta, om.zeta0, m.layer_thickness, op.OP_A)
        rng = np.random.default_rng(nz)
        xs = [_sources(m, nz, rng, kind), _sources(m, nz, rng, "falling")]
        apply = egx_ctx.op_apply if entry == "c128" else egx_ctx.op_apply_ds
        y = apply(np.concatenate(xs), nrhs=2).reshape(2, -1)
        for i in range(2):
            err = _layer_errors(y[i], op.apply(G, om, xs[i], op.OP_A), m, nz)
            assert err.max() < 4e-14, (i, err)
    finally:
        g.free()


def test_subnormal_vector_in_complex128(egx_ctx):
    """2^-1040 times a vector gives 2^-1040 times the result, to what rounding
    to units of 2^-1074 leaves: half a unit in each of ten steps, summed over
    120 spectral points by an operator of norm below three, 1,800 units."""
    nz = 9
    m, om, G = _case(egx_ctx, nz, 0.1, nz)
    g = egx_ctx.green_upload(G, m.nx, m.ny, nz)
    try:
        egx_ctx.op_prepare(g, om.zeta, om.zeta0, m.layer_thickness, op.OP_A)
        rng = np.random.default_rng(1)
        x = rng.standard_normal(m.nx * m.ny * 3 * nz) + 1j * rng.standard_normal(m.nx * m.ny * 3 * nz)
        y, small = egx_ctx.op_apply(x), egx_ctx.op_apply(np.ldexp(x.real, -1040) + 1j * np.ldexp(x.imag, -1040))
        d = np.ldexp(small.real, 1040) + 1j * np.ldexp(small.imag, 1040) - y
        assert np.abs(d).max() < 1800 * 2.0 ** (1040 - 1074)
    finally:
        g.free()


@pytest.mark.parametrize("nz,f", [(9, 0.1), (22, 0.1), (24, 10.0), (35, 1.0), (47, 0.1)])
@pytest.mark.parametrize("kind", ["one layer", "falling"])
def test_every_layer_in_complex64(egx_ctx, nz, f, kind):
    """The packed layouts, one and two right-hand sides."""
    m, om, G = _case(egx_ctx, nz, f, nz)
    g = egx_ctx.green_upload(G, m.nx, m.ny, nz, precision=egx.PREC_MIXED)
    try:
        egx_ctx.op_prepare(g, om.zeta, om.zeta0, m.layer_thickness, op.OP_A)
        rng = np.random.default_rng(nz)
        xs = [_sources(m, nz, rng, kind).astype(np.complex64), _sources(m, nz, rng, "falling").astype(np.complex64)]
        for nrhs in (1, 2):
            y = egx_ctx.op_apply_c64(np.concatenate(xs[:nrhs]), nrhs=nrhs).reshape(nrhs, -1)
            for i in range(nrhs):
                err = _layer_errors(y[i], op.apply(G, om, xs[i].astype(complex), op.OP_A), m, nz)
                assert err.max() < 2.2e-6, (nrhs, i, err)
    finally:
        g.free()


@pytest.mark.parametrize("nz", [16, 32, 48])
def test_every_layer_of_one_source_in_the_subblock_layout(egx_ctx, nz):
    """Layers without coupling: each one's response is its own source's, of
    whatever size that is beside the others."""
    m, om, G = _case(egx_ctx, nz, 0.1, nz)
    tr, rc = np.meshgrid(np.arange(nz), np.arange(nz), indexing="ij")
    up = rc <= tr
    G = {c: v * ((rc == tr).reshape(-1) if c in ("xz", "yz") else (rc == tr)[up]) for c, v in G.items()}
    g = egx_ctx.green_upload(G, m.nx, m.ny, nz, precision=egx.PREC_MIXED)
    try:
        egx_ctx.op_prepare(g, om.zeta, om.zeta0, m.layer_thickness, op.OP_A)
        x = _sources(m, nz, np.random.default_rng(nz), "falling").astype(np.complex64)
        err = _layer_errors(egx_ctx.op_apply_c64(x), op.apply(G, om, x.astype(complex), op.OP_A), m, nz)
        assert err.max() < 2e-5, err
    finally:
        g.free()


@pytest.mark.parametrize("nz", [9, 16, 32])
def test_one_complex64_source_keeps_what_is_not_finite(egx_ctx, nz):
    m, om, G = _case(egx_ctx, nz, 0.1, nz)
    g = egx_ctx.green_upload(G, m.nx, m.ny, nz, precision=egx.PREC_MIXED)
    try:
        egx_ctx.op_prepare(g, om.zeta, om.zeta0, m.layer_thickness, op.OP_A)
        x = np.ones(m.nx * m.ny * 3 * nz, np.complex64)
        assert np.isfinite(egx_ctx.op_apply_c64(x)).all()
        for bad in (np.nan, np.inf, 1j * np.inf):
            xb = x.copy()
            xb[len(x) // 2] = bad
            assert not np.isfinite(egx_ctx.op_apply_c64(xb)).any()
    finally:
        g.free()
