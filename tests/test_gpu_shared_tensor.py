"""GPU: a tensor is read-only once it is made. Contexts on several host threads
apply one tensor at the same time, and an operator takes no device memory
beside the tensor's own and the apply's buffers."""
import threading

import numpy as np
import pytest

from extreme_gb300 import egx
from extreme_gb300.model import OmegaModel, freq_to_omega, random_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,precision", [(16, egx.PREC_MIXED), (9, egx.PREC_MIXED), (12, egx.PREC_FP64)])
def test_contexts_share_a_tensor(egx_ctx, nz, precision):
    m = random_model(12, 10, nz, seed=nz)
    f = m.frequencies[1]
    om = OmegaModel.build(m, f)
    n = m.nx * m.ny * 3 * nz
    rng = np.random.default_rng(nz)
    xs = rng.standard_normal((4, n)) + 1j * rng.standard_normal((4, n))
    g = egx_ctx.green_build(m, freq_to_omega(f), 10, precision)
    contexts = [egx.Context(0) for _ in range(4)]
    out, errors = [[] for _ in contexts], []
    try:
        for ctx in contexts:
            ctx.op_prepare(g, om.zeta, om.zeta0, m.layer_thickness, egx.OP_A)
        start = threading.Barrier(len(contexts))

        def work(i):
            try:
                start.wait()
                for _ in range(3):
                    out[i].append(contexts[i].op_apply(xs[i]))
            except Exception as e:
                errors.append(e)

        threads = [threading.Thread(target=work, args=(i,)) for i in range(len(contexts))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors
        egx_ctx.op_prepare(g, om.zeta, om.zeta0, m.layer_thickness, egx.OP_A)
        for i in range(len(contexts)):
            want = egx_ctx.op_apply(xs[i])
            assert all(np.array_equal(y, want) for y in out[i]), i
    finally:
        for ctx in contexts:
            ctx.close()
        g.free()


@pytest.mark.parametrize("precision", [egx.PREC_FP64, egx.PREC_MIXED])
def test_a_tensor_takes_its_own_memory(precision):
    """48x48x22: 78 MB in complex128, half of it more in complex64."""
    torch = pytest.importorskip("torch")
    nx = ny = 48
    nz = 22
    blk = {c: nz * nz if c in ("xz", "yz") else nz * (nz + 1) // 2 for c in ("xx", "xy", "yy", "zz", "xz", "yz")}
    G = {c: np.zeros((2 * nx, 2 * ny, k), np.complex128) for c, k in blk.items()}
    tensor = (nx + 1) * (ny + 1) * 4 * nz * (nz + 1) * (16 if precision == egx.PREC_FP64 else 24)
    n = nx * ny * 3 * nz
    vectors = 16 * n * (3 + 4)  # staged vectors, transform buffer
    slack = 32 << 20  # the driver's pools
    ctx = egx.Context(0)
    try:
        ctx.fft2d(np.zeros((8, 8, 1), complex), -1)
        free0 = torch.cuda.mem_get_info(0)[0]
        g = ctx.green_upload(G, nx, ny, nz, precision=precision)
        free1 = torch.cuda.mem_get_info(0)[0]
        assert free0 - free1 < tensor + slack
        zeta = np.ones((nx, ny, nz), complex)
        ctx.op_prepare(g, zeta, np.ones(nz, complex), np.ones(nz), egx.OP_A)
        ctx.op_apply(np.ones(n, complex))
        assert free1 - torch.cuda.mem_get_info(0)[0] < 3 * vectors + slack
        g.free()
    finally:
        ctx.close()
