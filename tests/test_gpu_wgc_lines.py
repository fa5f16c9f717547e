"""The Wang-Govind-Carter term on every kind of grid line (GPU): its fields
ride the line passes of the rest of the functional, are combined along axis 0
and end in one pointwise epilogue; lines of one stage or with a prime factor
above 7 take passes of their own.

Reference: the expansion written out in numpy FP64 from the device's own four
kernel fields, with Thomas-Fermi and Hartree terms beside it.  Tolerance:
transforms of N points there and back err below 8 eps log2 N of their largest
value (eps = 2^-53 or 2^-24), powers and products below 16 eps; both are
weighed with the sum of the magnitudes of the terms.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(24, 28, 18), (27, 25, 21), (9, 2, 6), (216, 16, 20), (300, 10, 6), (360, 8, 12), (16, 36, 128),   # combined
         (8, 16, 24), (22, 12, 18), (512, 6, 10)]                                                           # their own


@pytest.mark.parametrize("prec", [1, 0])
@pytest.mark.parametrize("two", [True, False])
@pytest.mark.parametrize("base", [True, False])
@pytest.mark.parametrize("nr", GRIDS)
def test_wgc_on_lines(nr, base, two, prec):
    import torch
    from dftpy_gb300 import _lib
    from dftpy_gb300.functional.wgc import kernel_table
    _lib.require_cuda()
    a, b = (1.2, 0.47) if two else (5 / 6, 5 / 6)
    lat = np.diag([0.4 * k for k in nr])
    N, dV = int(np.prod(nr)), 0.4 ** 3
    dt = torch.float64 if prec else torch.float32
    rng = np.random.default_rng(N)
    rho = (0.03 + 0.01 * rng.random(nr)).astype(np.float64 if prec else np.float32).astype(np.float64)
    r0 = float(rho.mean())
    lib, L, s = _lib, _lib.load(), _lib.stream_ptr()
    plan = lib.Plan(nr, lat, precision=prec)
    nb = ctypes.c_int64()
    lib.check(L.gbofdft_wgc_workspace_bytes(plan.handle, ctypes.byref(nb)))
    buf = torch.empty(int(nb.value) // 8 + 64, dtype=torch.float64, device="cuda")
    K = torch.empty((4, nr[0], nr[1], nr[2] // 2 + 1), dtype=dt, device="cuda")
    t0, h, cols = kernel_table(a, b, 2.7, 1.0, 2)
    tab = torch.tensor(np.ascontiguousarray(cols), dtype=torch.float64, device="cuda")
    lib.check(L.gbofdft_wgc_kernels(plan.handle, r0, a, b, lib.ptr(tab), int(cols.shape[1]), t0, h, lib.ptr(K), s))
    d = lib.Wgc()
    d.alpha, d.beta, d.gamma, d.rho0, d.order = a, b, 2.7, r0, 2
    d.kernels, d.work, d.work_bytes = K.data_ptr(), lib.aligned_ptr(buf, 256), int(nb.value)
    f = lib.Functional()
    f.wgc = ctypes.pointer(d)
    if base:
        f.tf, f.tf_x, f.hartree = 1, 1.0, 1
    rd = torch.tensor(rho, dtype=dt, device="cuda")
    pot = torch.full(nr, float("nan"), dtype=dt, device="cuda")
    en = torch.zeros(lib.NE, dtype=torch.float64, device="cuda")
    lib.check(L.gbofdft_eval(plan.handle, lib.ptr(rd), f, lib.ptr(pot), lib.ptr(en), lib.CALC_E | lib.CALC_V, s))
    pv = torch.full(nr, float("nan"), dtype=dt, device="cuda")
    lib.check(L.gbofdft_eval(plan.handle, lib.ptr(rd), f, lib.ptr(pv), None, lib.CALC_V, s))
    torch.cuda.synchronize()

    K0, K1, Kq, Kx = K.double().cpu().numpy()
    u = (rho - r0) / r0
    size = 0.0

    def conv(k, x):
        nonlocal size
        y = np.fft.irfftn(k * np.fft.rfftn(x), s=nr, axes=(0, 1, 2))
        size = max(size, np.abs(k).max() * np.sqrt((x * x).mean()))
        return y

    def half(e):
        w = rho ** e
        return conv(K0, w) + conv(K1, u * w) / 6 + conv(Kq, u * u * w), conv(K1, w) / 6 + conv(Kx, u * w), conv(Kq, w)

    def add(x, e):
        return (e * rho ** (e - 1) * (x[0] + u * x[1] + u * u * x[2])
                + rho ** e / r0 * (x[1] + 2 * u * x[2]))

    X, Y = half(b), half(a)
    ref = add(X, a) + add(Y, b)
    e_nl = (rho ** a * (X[0] + u * X[1] + u * u * X[2])).sum() * dV
    # largest value of a term of V: d(rho^e) times an output
    scale = 6 * size * max(a * rho.max() ** (a - 1), b * rho.min() ** (b - 1))
    e_tot, e_size = e_nl, size * (rho ** a).sum() * dV
    if base:
        ctf = 0.3 * (3 * np.pi ** 2) ** (2 / 3)
        fr = [2 * np.pi * np.fft.fftfreq(n, d=0.4) for n in nr]
        gg = fr[0][:, None, None] ** 2 + fr[1][None, :, None] ** 2 + (fr[2][:nr[2] // 2 + 1] ** 2)[None, None, :]
        gg[0, 0, 0] = 1.0
        kh = 4 * np.pi / gg
        kh[0, 0, 0] = 0.0
        vh = np.fft.irfftn(kh * np.fft.rfftn(rho), s=nr, axes=(0, 1, 2))
        ref = ref + 5 / 3 * ctf * rho ** (2 / 3) + vh
        e_tot += ctf * (rho ** (5 / 3)).sum() * dV + 0.5 * (vh * rho).sum() * dV
        scale += 5 / 3 * ctf * rho.max() ** (2 / 3) + kh.max() * rho.max()
        e_size += abs(e_tot) + kh.max() * rho.max() * rho.sum() * dV
    eps = 2.0 ** -53 if prec else 2.0 ** -24
    tol = (8 * np.log2(N) + 16) * eps
    assert np.abs(pot.double().cpu().numpy() - ref).max() <= tol * scale
    assert np.abs(pv.double().cpu().numpy() - ref).max() <= tol * scale
    assert abs(float(en[lib.E_NL]) - e_nl) <= tol * e_size
    assert abs(float(en[lib.E_TOTAL]) - e_tot) <= tol * e_size


def test_wgc_beside_the_plane_pipeline():
    """A plan set to the plane schedule: the other terms on planes, the WGC term on
    lines, added; the same potential and energies as on lines alone within the FP32
    bound above."""
    import torch
    from dftpy_gb300 import _lib as lib
    from dftpy_gb300.functional.wgc import kernel_table
    lib.require_cuda()
    nr, N = (64, 64, 32), 64 * 64 * 32
    L, s = lib.load(), lib.stream_ptr()
    plan = lib.Plan(nr, np.diag([0.4 * k for k in nr]), precision=0)
    rho = 0.03 + 0.01 * np.random.default_rng(1).random(nr)
    r0 = float(rho.mean())
    nb = ctypes.c_int64()
    lib.check(L.gbofdft_wgc_workspace_bytes(plan.handle, ctypes.byref(nb)))
    buf = torch.empty(int(nb.value) // 8 + 64, dtype=torch.float64, device="cuda")
    K = torch.empty((4, 64, 64, 17), dtype=torch.float32, device="cuda")
    t0, h, cols = kernel_table(1.2, 0.47, 2.7, 1.0, 2)
    tab = torch.tensor(np.ascontiguousarray(cols), dtype=torch.float64, device="cuda")
    lib.check(L.gbofdft_wgc_kernels(plan.handle, r0, 1.2, 0.47, lib.ptr(tab), int(cols.shape[1]), t0, h, lib.ptr(K), s))
    d = lib.Wgc()
    d.alpha, d.beta, d.gamma, d.rho0, d.order = 1.2, 0.47, 2.7, r0, 2
    d.kernels, d.work, d.work_bytes = K.data_ptr(), lib.aligned_ptr(buf, 256), int(nb.value)
    f = lib.Functional()
    f.wgc = ctypes.pointer(d)
    f.tf, f.tf_x, f.hartree = 1, 1.0, 1
    rd = torch.tensor(rho, dtype=torch.float32, device="cuda")
    res = []
    for sched in (0, 1):
        lib.check(L.gbofdft_plan_set_schedule(plan.handle, sched))
        pot = torch.full(nr, float("nan"), dtype=torch.float32, device="cuda")
        en = torch.zeros(lib.NE, dtype=torch.float64, device="cuda")
        lib.check(L.gbofdft_eval(plan.handle, lib.ptr(rd), f, lib.ptr(pot), lib.ptr(en), lib.CALC_E | lib.CALC_V, s))
        res.append((pot.double().cpu().numpy(), en.cpu().numpy()))
    tol = (8 * np.log2(N) + 16) * 2.0 ** -24
    (p0, e0), (p1, e1) = res
    # |4 pi / G^2| rho is the largest term
    scale = 4 * np.pi / (2 * np.pi / (0.4 * 64)) ** 2 * rho.max()
    assert np.abs(p0 - p1).max() <= tol * scale
    assert np.abs(e0 - e1).max() <= tol * scale * rho.sum() * 0.4 ** 3
