"""GPU: what a context keeps between calls (FFT tables, term lists, operator)
after a call that ran out of device memory half way, at each of its
allocations in turn. The failure is made on the host (an allocation that is
refused); afterwards the call of before gives what it gave before, bit for
bit, or says that there is no operator."""
import numpy as np
import pytest

from extreme_gb300 import egx
from extreme_gb300.model import OmegaModel, freq_to_omega, random_model

pytestmark = pytest.mark.gpu
F = 0.3


def _build(precision):
    def call(ctx, m):
        g = ctx.green_build(m, freq_to_omega(F), 10, precision)
        G = g.download()
        om = OmegaModel.build(m, F)
        ctx.op_prepare(g, om.zeta, om.zeta0, m.layer_thickness, egx.OP_A)
        x = np.ones(m.nx * m.ny * 3 * m.nz, complex)
        y = [ctx.op_apply(x)]
        if precision == egx.PREC_MIXED:
            y.append(ctx.op_apply_c64(x))
        g.free()
        return [G[c] for c in sorted(G)] + y
    return call


def _level(precision):
    def call(ctx, m):
        n = m.nx * m.ny * 3 * m.nz
        ctx.level_cache(0)
        return list(ctx.level_fields(m, freq_to_omega(F), np.ones((1, n), complex), precision=precision))
    return call


@pytest.mark.parametrize("call,a,b", [(_build(egx.PREC_FP64), (12, 10, 3), (20, 18, 4)),
                                      (_build(egx.PREC_MIXED), (32, 32, 3), (64, 32, 4)),
                                      (_level(egx.PREC_FP64), (12, 10, 3), (20, 18, 4)),
                                      (_level(egx.PREC_MIXED), (32, 32, 3), (64, 32, 4))],
                         ids=["build64", "build32", "level64", "level32"])
def test_the_call_after_one_without_memory(call, a, b):
    ma, mb = random_model(*a, seed=1), random_model(*b, seed=2)
    failures = 0
    for n in range(1, 200):
        ctx = egx.Context(0)
        try:
            want = call(ctx, ma)
            ctx.inject_alloc_failure(n)
            try:
                call(ctx, mb)
            except egx.EgxError as e:
                assert e.code == egx.ERR_OOM
                failures += 1
            else:
                break
            finally:
                ctx.inject_alloc_failure(0)
            got = call(ctx, ma)
            assert all(np.array_equal(x, y) for x, y in zip(want, got)), n
        finally:
            ctx.close()
    assert failures >= 10


def test_no_operator_after_a_failed_preparation():
    ma, mb = random_model(12, 10, 3, seed=1), random_model(20, 18, 4, seed=2)
    ctx = egx.Context(0)
    try:
        ga, gb = (ctx.green_build(m, freq_to_omega(F)) for m in (ma, mb))
        om = OmegaModel.build(ma, F)
        ctx.op_prepare(ga, om.zeta, om.zeta0, ma.layer_thickness, egx.OP_A)
        om = OmegaModel.build(mb, F)
        ctx.inject_alloc_failure(3)
        with pytest.raises(egx.EgxError) as e:
            ctx.op_prepare(gb, om.zeta, om.zeta0, mb.layer_thickness, egx.OP_A)
        ctx.inject_alloc_failure(0)
        assert e.value.code == egx.ERR_OOM
        with pytest.raises(egx.EgxError) as e:
            ctx.op_apply(np.ones(ma.nx * ma.ny * 3 * ma.nz, complex))
        assert e.value.code == egx.ERR_STATE
        ga.free()
        gb.free()
    finally:
        ctx.close()
