"""What the framework's users have it do, as cases that can be timed.

The work is the integral-equation forward solve: operator applies (the inner
loop of every solve), the 2-D FFT, the Green tensor and first apply of a new
frequency, the fields at an observation level, whole forward solves, and a
training step of the learned preconditioner. Sizes are those of the
benchmark's configurations (32x32x8 plain small, 128x128x32 plain medium and
learned, 256x256x48 precision, uneven meshes between 64x64x16 and 192x160x40
batching) and generic ones in between.
"""
import math

import numpy as np
import torch

from extreme_gb300 import egx
from extreme_gb300.forward import ForwardSettings, MixedSettings, Mt3DForwardSolver, model_zeta
from extreme_gb300.model import EPS0, freq_to_omega, random_model, small_model

DEV = "cuda"
COMPS = ("xx", "xy", "yy", "zz", "xz", "yz")
MODES = 16  # retained lateral modes per direction of the learned network


def listed():
    return [
        # one step of the plain method's smallest configuration: five small
        # kernels and the host's share of a call
        {"name": "apply_c128_small", "kind": "apply", "prec": "c128", "nx": 32, "ny": 32, "nz": 8, "nrhs": 1},
        # the plain (reference) method's mat-vec at the medium configuration
        {"name": "apply_c128_medium", "kind": "apply", "prec": "c128", "nx": 128, "ny": 128, "nz": 32, "nrhs": 1},
        # the mixed form's residual apply, both polarisations
        {"name": "apply_ds_medium", "kind": "apply", "prec": "ds", "nx": 128, "ny": 128, "nz": 32, "nrhs": 2},
        # the mixed form's inner mat-vec, one polarisation at a time
        {"name": "apply_c64_medium", "kind": "apply", "prec": "c64", "nx": 128, "ny": 128, "nz": 32, "nrhs": 1},
        # the batching form's uneven meshes: odd depth, 7-smooth lateral sizes
        {"name": "apply_c64_uneven", "kind": "apply", "prec": "c64", "nx": 180, "ny": 120, "nz": 35, "nrhs": 2},
        # the precision form's inner mat-vec at full size, both polarisations
        {"name": "apply_c64_precision", "kind": "apply", "prec": "c64", "nx": 256, "ny": 256, "nz": 48, "nrhs": 2},
        # the FFT entry point on a medium spectral buffer (nz = 32, one source)
        {"name": "fft2d", "kind": "fft2d", "n0": 256, "n1": 256, "howmany": 96, "sign": -1},
        # a new frequency of the plain method: Green tensor, operator, first apply
        {"name": "frequency", "kind": "frequency", "nx": 128, "ny": 128, "nz": 32},
        # surface fields of both polarisations, level tensors built for the frequency
        {"name": "level_fields", "kind": "level", "nx": 128, "ny": 128, "nz": 32},
        # the whole plain forward solve of the small configuration
        {"name": "solve_plain_small", "kind": "solve", "prec": "fp64", "nx": 32, "ny": 32, "nz": 8},
        # the whole mixed forward solve of an uneven mesh, refined far enough
        # to be compared with the plain method's fields
        {"name": "solve_mixed_uneven", "kind": "solve", "prec": "mixed", "nx": 90, "ny": 75, "nz": 22},
        # one training step of the learned preconditioner (loss and gradient)
        {"name": "net_train", "kind": "net", "nx": 128, "ny": 128, "nz": 32, "batch": 8},
    ]


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def _lateral(rng, lo, hi):
    """A lateral size with a 7-smooth transform length, spread over the logarithm."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    while not _smooth(n) or n > hi:
        n -= 1
    return max(n, lo)


def _depth(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("apply",) * 6 + ("fft2d", "frequency", "level", "solve", "net"))
    if kind == "apply":
        return {"kind": kind, "prec": rng.choice(("c64", "c64", "c128", "c128", "ds")), "nx": _lateral(rng, 16, 192),
                "ny": _lateral(rng, 16, 160), "nz": _depth(rng, 4, 48), "nrhs": rng.choice((1, 1, 2, 2, 3))}
    if kind == "fft2d":
        return {"kind": kind, "n0": _lateral(rng, 16, 512), "n1": _lateral(rng, 16, 512),
                "howmany": _depth(rng, 3, 144), "sign": rng.choice((-1, 1))}
    if kind in ("frequency", "level"):
        return {"kind": kind, "nx": _lateral(rng, 16, 128), "ny": _lateral(rng, 16, 128), "nz": _depth(rng, 4, 32)}
    if kind == "solve":
        if rng.random() < 0.5:
            return {"kind": kind, "prec": "fp64", "nx": _lateral(rng, 16, 40), "ny": _lateral(rng, 16, 40),
                    "nz": _depth(rng, 4, 12)}
        # uneven meshes, whose tensors the mixed form builds in 64 bits throughout
        return {"kind": kind, "prec": "mixed", "nx": _lateral(rng, 36, 90), "ny": rng.choice((45, 50, 63, 75)),
                "nz": _depth(rng, 9, 24)}
    return {"kind": kind, "nx": _lateral(rng, 32, 128), "ny": _lateral(rng, 32, 128), "nz": _depth(rng, 8, 32),
            "batch": rng.choice((1, 2, 3, 4, 8))}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _randn(shape, g, dtype=torch.complex128):
    return torch.randn(shape, generator=g, device=DEV, dtype=dtype)


def _layers(nz):
    th = np.round(100.0 * 1.1 ** np.arange(nz), 2)
    return np.concatenate([[0.0], np.cumsum(th)[:-1]]), th


def _medium(case, seed):
    """Layer thicknesses and conductivities of an operator: a layered
    background and boxes two decades up and down."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    depth, th = _layers(nz)
    omega = freq_to_omega(10.0 ** rng.uniform(-3, 1))
    bg = np.repeat(10.0 ** rng.uniform(-3, 0, nz // 4 + 1), 4)[:nz]
    sigma = np.broadcast_to(bg, (nx, ny, nz)).copy()
    for _ in range(20):
        x, y, z = rng.integers(0, nx), rng.integers(0, ny), rng.integers(0, nz)
        sigma[x:x + nx // 4 + 1, y:y + ny // 4 + 1, z:z + nz // 3 + 1] = 10.0 ** rng.uniform(-3, 0.5)
    return depth, th, omega, sigma - 1j * omega * EPS0, bg - 1j * omega * EPS0


def _green_quadrant(case, seed):
    """A spectral Green tensor of the reference's form on the stored quadrant:
    entries that decay with wavenumber times layer distance, sized so that the
    operator's scattering part is near the identity's size, over the rounding
    floor of a numerically transformed tensor."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = _gen(1000003 * seed + 17)
    depth, th, _, _, zeta0 = _medium(case, seed)
    z = torch.tensor(depth + th / 2, device=DEV)
    h = torch.tensor(th, device=DEV)
    s0 = torch.tensor(zeta0.real, device=DEV)
    step = 500.0
    kx = (math.pi / (nx * step)) * torch.arange(nx + 1, device=DEV, dtype=torch.float64)
    ky = (math.pi / (ny * step)) * torch.arange(ny + 1, device=DEV, dtype=torch.float64)
    k = torch.sqrt(kx[:, None] ** 2 + ky[None, :] ** 2 + 1e-8)[:, :, None]
    tr, rc = torch.meshgrid(torch.arange(nz, device=DEV), torch.arange(nz, device=DEV), indexing="ij")
    up = rc <= tr  # row-major over (tr, rc) is the packed order rc + tr(tr+1)/2
    pairs = {"sym": (rc[up], tr[up]), "all": (tr.reshape(-1), rc.reshape(-1))}
    out = {}
    for c in COMPS:
        i, j = pairs["all" if c in ("xz", "yz") else "sym"]
        fall = torch.exp(-k * (z[i] - z[j]).abs()) * (h[i] * h[j] * k / (1 + k * torch.sqrt(h[i] * h[j])))
        fall /= 4 * torch.sqrt(s0[i] * s0[j])
        floor = 1e-16 * fall.amax()
        wide = {"xx": kx[:, None, None] / k, "xy": 0.5 * kx[:, None, None] * ky[None, :, None] / k ** 2,
                "yy": ky[None, :, None] / k, "zz": torch.ones_like(k), "xz": 0.7 * kx[:, None, None] / k,
                "yz": 0.7 * ky[None, :, None] / k}[c]
        v = torch.empty((nx + 1, ny + 1, len(i)), dtype=torch.complex128, device=DEV)
        for a in range(0, nx + 1, 16):
            n = min(16, nx + 1 - a)
            r = _randn((n, ny + 1, len(i)), g)
            w = wide[a:a + n] if wide.shape[0] > 1 else wide
            v[a:a + n] = fall[a:a + n] * w * (1 + 0.2 * r) + floor * r.conj()
        out[c] = v
    return out


def _upload(ctx, case, seed, prec):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    host = {}
    for c, v in _green_quadrant(case, seed).items():
        full = np.zeros((2 * nx, 2 * ny, v.shape[2]), np.complex128)
        full[:nx + 1, :ny + 1] = v.cpu().numpy()
        host[c] = full
    return ctx.green_upload(host, nx, ny, nz, prec)


def _torch_ctx():
    """A context on the stream that torch works on."""
    ctx = egx.Context()
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    return ctx


def _vectors(case, seed, dtype):
    """Right-hand sides as a solve has them: Krylov vectors whose layers differ in size."""
    nx, ny, nz, nrhs = case["nx"], case["ny"], case["nz"], case.get("nrhs", 1)
    g = _gen(1000003 * seed + 29)
    amp = torch.exp(-torch.arange(nz, device=DEV, dtype=torch.float64) / (0.3 * nz + 1))
    x = _randn((nrhs, nx, ny, 3, nz), g) * amp
    x /= torch.linalg.vector_norm(x.reshape(nrhs, -1), dim=1).reshape(-1, 1, 1, 1, 1)
    return x.to(dtype).contiguous()


def _built(case):
    """Whether an apply's tensor is built from a layered model: in the
    reference's layout the largest ones do not fit the host."""
    return case["nx"] * case["ny"] * case["nz"] ** 2 > 192 * 160 * 48 ** 2


def _model(case, seed):
    return random_model(case["nx"], case["ny"], case["nz"], seed=seed % 100000)


def _frequency(seed):
    return float(10.0 ** np.random.default_rng(seed + 5).uniform(-2, 0))


def prepare(case, seed):
    state = globals()["_prepare_" + case["kind"]](case, seed)
    torch.cuda.synchronize()
    return state


def _prepare_apply(case, seed):
    ctx = _torch_ctx()
    prec = egx.PREC_FP64 if case["prec"] == "c128" else egx.PREC_MIXED
    dtype = torch.complex64 if case["prec"] == "c64" else torch.complex128
    if _built(case):
        model = _model(case, seed)
        omega = freq_to_omega(_frequency(seed))
        green = ctx.green_build(model, omega, 10, prec)
        zeta, zeta0 = model_zeta(model, omega)
        dz = model.layer_thickness
    else:
        _, dz, _, zeta, zeta0 = _medium(case, seed)
        green = _upload(ctx, case, seed, prec)
    ctx.op_prepare(green, zeta, zeta0, dz, egx.OP_A)
    x = _vectors(case, seed, dtype)
    return {"kind": "apply", "prec": case["prec"], "ctx": ctx, "green": green, "nrhs": case["nrhs"], "x": x,
            "y": torch.empty_like(x)}


def _prepare_fft2d(case, seed):
    x = _randn((case["n0"], case["n1"], case["howmany"]), _gen(1000003 * seed + 31))
    return {"kind": "fft2d", "ctx": _torch_ctx(), "x": x, "buf": torch.empty_like(x), "sign": case["sign"]}


def _prepare_frequency(case, seed):
    model = _model(case, seed)
    f = _frequency(seed)
    zeta, zeta0 = model_zeta(model, freq_to_omega(f))
    x = _vectors(case, seed, torch.complex128)
    return {"kind": "frequency", "ctx": _torch_ctx(), "model": model, "omega": freq_to_omega(f), "zeta": zeta,
            "zeta0": zeta0, "x": x, "y": torch.empty_like(x)}


def _prepare_level(case, seed):
    model = _model(case, seed)
    ctx = _torch_ctx()
    ctx.level_cache(0)  # every frequency is a new one
    jq = _vectors(dict(case, nrhs=2), seed, torch.complex128)
    e = torch.empty((2, case["nx"], case["ny"], 3), dtype=torch.complex128, device=DEV)
    return {"kind": "level", "ctx": ctx, "model": model, "omega": freq_to_omega(_frequency(seed)), "jq": jq, "e": e,
            "h": torch.empty_like(e)}


def _prepare_solve(case, seed):
    rng = np.random.default_rng(seed)
    if case["prec"] == "fp64":
        if (case["nx"], case["ny"], case["nz"]) == (32, 32, 8):
            model, f = small_model(), 0.1
            model.sigma[15:17, 15:17, :] *= rng.uniform(0.5, 2.0)  # the cube of the small configuration
        else:
            model, f = _model(case, seed), 0.1
        solver = Mt3DForwardSolver(ForwardSettings(residual=1e-8, outer_buffer_length=20))
        levels = (0.0,)
    else:
        model, f = _model(case, seed), _frequency(seed)
        solver = Mt3DForwardSolver(precision=egx.PREC_MIXED, mixed=MixedSettings(tol=1e-10))
        levels = ()
    return {"kind": "solve", "solver": solver, "model": model, "f": f, "levels": levels}


def _net_sizes(case, width=32, layers=4):
    nz, W = case["nz"], width
    sizes = [("P", (7, W)), ("bP", (W,))]
    for l in range(layers):
        sizes += [("Wm%d" % l, (MODES * MODES, W, W)), ("Wp%d" % l, (W, W)), ("Dz%d" % l, (nz, nz)), ("b%d" % l, (W,))]
    return sizes + [("Q", (W, 6)), ("bQ", (6,))]


def _net_params(case, seed):
    """Parameters of a network some way into its training."""
    rng = np.random.default_rng(seed + 71)
    out = {}
    for name, shape in _net_sizes(case):
        sd = {"P": 7 ** -0.5, "W": 1 / 32 if name[1:2] == "m" else 32 ** -0.5, "D": 0.5 * case["nz"] ** -0.5,
              "Q": 0.1 * 32 ** -0.5, "b": 0.02}[name[0]]
        out[name] = (sd * rng.standard_normal(shape)).astype(np.float32)
    return out


def _net_inputs(case, seed):
    nx, ny, nz, b = case["nx"], case["ny"], case["nz"], case["batch"]
    v = _vectors(dict(case, nrhs=b), seed, torch.complex64).reshape(b, -1)
    t = (0.2 * v + 0.3 * _vectors(dict(case, nrhs=b), seed + 7919, torch.complex64).reshape(b, -1)).contiguous()
    rng = np.random.default_rng(seed + 3)
    logsig = rng.uniform(-3, 1, (b, (nx + 7) // 8, (ny + 7) // 8, nz)).repeat(8, 1).repeat(8, 2)[:, :nx, :ny]
    return v, t, np.ascontiguousarray(logsig, np.float32)


def _prepare_net(case, seed):
    ctx = _torch_ctx()
    net = egx.SpectralNet(ctx, case["nx"], case["ny"], case["nz"], width=32, layers=4, seed=seed % 100000)
    flat = []
    for a in _net_params(case, seed).values():
        flat += [a.reshape(-1), np.zeros(-a.size % 4, np.float32)]
    net.params(np.concatenate(flat))
    v, t, logsig = _net_inputs(case, seed)
    net.set_model(logsig)
    return {"kind": "net", "ctx": ctx, "net": net, "v": v, "t": t, "batch": case["batch"]}


# --------------------------------------------------------------------- run
def run(state):
    return globals()["_run_" + state["kind"]](state)


def _run_apply(s):
    ctx, x, y = s["ctx"], s["x"], s["y"]
    if s["prec"] == "c128":
        ctx.op_apply_dev(x.data_ptr(), y.data_ptr(), s["nrhs"])
    else:
        entry = ctx.lib.egx_op_apply_c64 if s["prec"] == "c64" else ctx.lib.egx_op_apply_ds
        ctx._check(entry(ctx.h, x.data_ptr(), y.data_ptr(), s["nrhs"], egx.DEVICE))
    return y


def _run_fft2d(s):
    ctx, buf = s["ctx"], s["buf"]
    buf.copy_(s["x"])  # the transform is in place
    n0, n1, howmany = buf.shape
    ctx._check(ctx.lib.egx_fft2d(ctx.h, buf.data_ptr(), n0, n1, howmany, s["sign"], egx.DEVICE))
    return buf


def _run_frequency(s):
    ctx, model = s["ctx"], s["model"]
    green = ctx.green_build(model, s["omega"])
    ctx.op_prepare(green, s["zeta"], s["zeta0"], model.layer_thickness, egx.OP_A)
    ctx.op_apply_dev(s["x"].data_ptr(), s["y"].data_ptr())
    green.free()
    return s["y"]


def _run_level(s):
    s["ctx"].level_fields_dev(s["model"], s["omega"], s["jq"].data_ptr(), 2, s["e"].data_ptr(), s["h"].data_ptr())
    return s["e"], s["h"]


def _run_solve(s):
    sol = s["solver"].solve(s["model"], s["f"], levels=s["levels"])
    return [sol.jq] + [a for lv in sol.levels for a in (lv.e, lv.h, lv.impedance, lv.rho)]


def _run_net(s):
    ctx, loss = s["ctx"], egx.C.c_float()
    grad = np.empty(s["net"].size, np.float32)
    ctx._check(ctx.lib.egx_net_loss_grad(ctx.h, s["net"].h, s["v"].data_ptr(), s["t"].data_ptr(), s["batch"],
                                         egx.C.byref(loss), grad.ctypes.data, egx.DEVICE))
    return np.float32(loss.value), grad


# -------------------------------------------------------------------- work
def _apply_work(case, size, nrhs):
    """An apply: the stored quarter of the tensor, the vectors in and out, r;
    the zero-padded transforms both ways and the block products."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    entries = (nx + 1) * (ny + 1) * (2 * nz * (nz + 1) + 2 * nz * nz)
    vec = nx * ny * 3 * nz
    fft = 2 * 5 * 3 * nz * nrhs * (nx * 2 * ny * math.log2(2 * ny) + 4 * nx * ny * math.log2(2 * nx))
    return {"bytes": size * (entries + 2 * nrhs * vec + vec // 3), "flops": 8 * 9 * nz * nz * 4 * nx * ny * nrhs + fft}


def work(case):
    kind = case["kind"]
    if kind == "apply":
        # the tensor in the precision that the form keeps: complex128, or complex64
        return _apply_work(case, 8 if case["prec"] == "c64" else 16, case["nrhs"])
    if kind == "fft2d":
        n = case["n0"] * case["n1"] * case["howmany"]
        return {"bytes": 32 * n, "flops": 5 * n * math.log2(case["n0"] * case["n1"])}
    nx, ny = case["nx"], case["ny"]
    if kind == "frequency":
        # the tensor written, read by the apply; its transform from the quadrant
        w = _apply_work(case, 16, 1)
        e = case["nz"] * (case["nz"] + 1) * 2 + 2 * case["nz"] ** 2
        fft = 5 * e * (nx * 2 * ny * math.log2(2 * ny) + (ny + 1) * 2 * nx * math.log2(2 * nx))
        return {"bytes": w["bytes"] + 16 * (nx + 1) * (ny + 1) * e, "flops": w["flops"] + fft}
    if kind == "level":
        nz, n = case["nz"], 4 * nx * ny
        fft = 5 * math.log2(n) * n * nz
        return {"bytes": 16 * (2 * 3 * nx * ny * nz + 2 * 2 * 3 * nx * ny + 2 * 15 * n * nz),
                "flops": fft * (15 + 6) + 2 * n * nz * 17 * 8}
    if kind == "solve":
        # about what the method needs in applies at these sizes, and the tensor
        applies, nrhs, size = (90, 1, 16) if case["prec"] == "fp64" else (220, 2, 8)
        w = _apply_work(case, size, nrhs)
        return {"bytes": applies * w["bytes"], "flops": applies * w["flops"]}
    nz, b, W = case["nz"], case["batch"], 32
    rows = b * nz * nx * ny
    per = 2 * (7 * W + 6 * W + 4 * (W * W + nz * W + 2 * MODES * W))  # multiply-adds of a row, forward
    par = 4 * (MODES * MODES * W * W + W * W + nz * nz)
    return {"bytes": 16 * rows * 3 + 4 * rows * W * 4 * 2 + 8 * par, "flops": 3 * per * rows}


# ------------------------------------------------------------------- exact
def _sym_dense(p, nz):
    """[..., nz(nz+1)/2] packed rc + tr(tr+1)/2 -> [..., nz, nz]."""
    i = torch.arange(nz, device=DEV)
    lo, hi = torch.minimum(i[:, None], i[None, :]), torch.maximum(i[:, None], i[None, :])
    return p[..., lo + hi * (hi + 1) // 2]


def _exact_apply(case, seed):
    if _built(case):
        return None  # its tensor is what the framework builds
    nx, ny, nz, nrhs = case["nx"], case["ny"], case["nz"], case["nrhs"]
    _, dz, _, zeta, zeta0 = _medium(case, seed)
    q = _green_quadrant(case, seed)
    dtype = torch.complex64 if case["prec"] == "c64" else torch.complex128
    x = _vectors(case, seed, dtype).to(torch.complex128)
    zeta, zeta0 = torch.tensor(zeta, device=DEV), torch.tensor(zeta0, device=DEV)
    dz = torch.tensor(dz, device=DEV)
    r = ((zeta - zeta0) / (zeta + zeta0.conj()))[:, :, None, :]
    root = torch.sqrt(zeta0.real)
    rx = r * x
    f = torch.fft.fft2(root * rx, s=(2 * nx, 2 * ny), dim=(1, 2))
    ky = torch.arange(2 * ny, device=DEV)
    b, my = torch.where(ky <= ny, ky, 2 * ny - ky), torch.where(ky <= ny, 1.0, -1.0).to(torch.float64)
    for kx in range(2 * nx):
        a, mx = (kx, 1.0) if kx <= nx else (2 * nx - kx, -1.0)
        sx, sy = mx, my[:, None, None]
        xx, yy, zz = (_sym_dense(q[c][a, b], nz) for c in ("xx", "yy", "zz"))
        xy = _sym_dense(q["xy"][a, b], nz) * (sx * sy)
        xz = q["xz"][a, b].reshape(-1, nz, nz) * sx
        yz = q["yz"][a, b].reshape(-1, nz, nz) * sy
        m = torch.cat([torch.cat([xx, xy, xz], 2), torch.cat([xy, yy, yz], 2),
                       torch.cat([-xz.transpose(1, 2), -yz.transpose(1, 2), zz], 2)], 1)
        v = f[:, kx].reshape(nrhs, 2 * ny, 3 * nz).permute(1, 2, 0)
        f[:, kx] = torch.bmm(m, v).permute(2, 0, 1).reshape(nrhs, 2 * ny, 3, nz)
    back = torch.fft.ifft2(f, dim=(1, 2))[:, :nx, :ny] * (2 * root / dz)
    return x - back - rx


def _exact_fft2d(case, seed):
    x = _randn((case["n0"], case["n1"], case["howmany"]), _gen(1000003 * seed + 31))
    if case["sign"] < 0:
        return torch.fft.fft2(x, dim=(0, 1))
    return torch.fft.ifft2(x, dim=(0, 1)) * (case["n0"] * case["n1"])


def _exact_net(case, seed):
    nx, ny, nz, B = case["nx"], case["ny"], case["nz"], case["batch"]
    v, t, logsig = _net_inputs(case, seed)
    p = {k: torch.tensor(a, device=DEV, dtype=torch.float64, requires_grad=True)
         for k, a in _net_params(case, seed).items()}

    def basis(n):
        i = torch.arange(n, device=DEV, dtype=torch.float64)[:, None] * (2 * math.pi / n)
        b = torch.cat([torch.cos(i * torch.arange(8, device=DEV)), torch.sin(i * torch.arange(1, 9, device=DEV))], 1)
        norm = torch.linalg.vector_norm(b, dim=0)
        return torch.where(norm > 1e-9, b / norm.clamp_min(1e-30), 0.0).to(torch.float32).double()

    bx, by = basis(nx), basis(ny)

    def planes(u):  # [nx][ny][3][nz] -> [nz][nx][ny][6]
        u = u.to(torch.complex128).reshape(nx, ny, 3, nz).permute(3, 0, 1, 2)
        return torch.cat([u.real, u.imag], 3)

    loss = torch.zeros((), device=DEV, dtype=torch.float64)
    for b in range(B):
        rms = torch.sqrt(v[b].to(torch.complex128).abs().square().mean())
        sig = torch.tensor(logsig[b], device=DEV, dtype=torch.float64).permute(2, 0, 1)[..., None]
        H = torch.cat([planes(v[b]) / rms, sig], 3) @ p["P"] + p["bP"]
        for l in range(4):
            U = torch.einsum("zxyc,xk,yl->zklc", H, bx, by)
            V = torch.einsum("zklc,klcd->zkld", U, p["Wm%d" % l].reshape(MODES, MODES, 32, 32))
            pre = torch.einsum("zklc,xk,yl->zxyc", V, bx, by) + H @ p["Wp%d" % l]
            pre = pre + torch.einsum("zw,wxyc->zxyc", p["Dz%d" % l], H) + p["b%d" % l]
            H = torch.nn.functional.gelu(pre, approximate="tanh") if l < 3 else pre
        target = planes(t[b]) / rms
        part = ((H @ p["Q"] + p["bQ"] - target) ** 2).sum() / (target ** 2).sum() / B
        part.backward()
        loss = loss + part.detach()
    flat = []
    for a in p.values():
        flat += [a.grad.reshape(-1), torch.zeros(-a.numel() % 4, device=DEV, dtype=torch.float64)]
    return loss, torch.cat(flat)


def exact(case, seed):
    """The applies, the FFT and the network in 64 bits. None for the rest:
    their tensors come from the layered earth's filtered integrals, which
    plain torch or numpy does not have within the time."""
    made = globals().get("_exact_" + case["kind"])
    return made(case, seed) if made else None
