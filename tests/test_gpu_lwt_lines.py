"""Batched knots of the LWT / LMGP term (GPU) against the same term written out
in numpy FP64: fewer knots than a batch, whole and partial batches, points below
the first knot and on every interval; lines of one stage and with a prime factor
above 7 take the passes of one knot at a time.

Tolerance: transforms of N points err below 8 eps log2 N of their largest value
(eps = 2^-53 or 2^-24), the cubic look-ups and powers below 32 eps; both are
weighed with the sum of the magnitudes of a point's terms.  FP32 look-ups read
coefficients rounded to FP32 on cells of 1/1000: another 2 eps of the kernel.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [((24, 28, 18), 1.15, 3), ((27, 25, 21), 1.15, 3), ((216, 6, 20), 1.3, 3), ((12, 10, 360), 2.0, 3),
         ((9, 2, 6), 1.05, 3), ((20, 18, 16), 1.15, 2), ((20, 18, 16), 1.15, 1), ((30, 11, 12), 1.15, 3),
         ((8, 12, 10), 1.15, 3)]


@pytest.mark.parametrize("prec", [1, 0])
@pytest.mark.parametrize("nr,ratio,kdd", CASES)
def test_lwt_batches(nr, ratio, kdd, prec):
    import torch
    from dftpy_gb300 import _lib as lib
    from dftpy_gb300._tables import spline_notaknot
    lib.require_cuda()
    h = 0.4
    lat = np.diag([h * k for k in nr])
    N, dV = int(np.prod(nr)), h ** 3
    dt = torch.float64 if prec else torch.float32
    rng = np.random.default_rng(N)
    rho = 0.002 + 0.05 * rng.random(nr) ** 3
    rho = (rho if prec else rho.astype(np.float32)).astype(np.float64)
    # a smooth stand-in for the kernel table
    etamax, neta = 30.0, 4001
    eta = np.linspace(0, etamax, neta)
    x, kc = spline_notaknot(eta, eta ** 2 / (1 + eta ** 2) - 0.3 * np.exp(-eta))
    _, dc = spline_notaknot(eta, np.cos(eta) * np.exp(-0.2 * eta))
    kd, dd = (torch.tensor(c.reshape(-1), dtype=torch.float64, device="cuda") for c in (kc, dc))
    d = lib.Lwt()
    d.interp, d.kdd, d.alpha, d.beta, d.ratio, d.ldw = 0, kdd, 5 / 6, 5 / 6, ratio, 0.0
    d.etamax, d.neta = etamax, neta
    kf = 2.0 * np.cbrt(3.0 * np.pi ** 2 * rho)
    d.kfmin_opt, d.kfmax_opt = 1.1 * kf.min(), 0.97 * kf.max()       # points below and above the knots
    d.kfmin_state = d.kfmax_state = 0.0
    d.ktab_c, d.dtab_c = kd.data_ptr(), dd.data_ptr()
    fk = eta[-1] ** 2 / (1 + eta[-1] ** 2) - 0.3 * np.exp(-eta[-1])
    fd = np.cos(eta[-1]) * np.exp(-0.2 * eta[-1])
    d.ktab_end, d.dtab_end = fk, fd
    L, s = lib.load(), lib.stream_ptr()
    plan = lib.Plan(nr, lat, precision=prec)
    nb = ctypes.c_int64()
    lib.check(L.gbofdft_lwt_workspace_bytes(plan.handle, ctypes.byref(nb)))
    buf = torch.full((int(nb.value) // 8 + 64,), float("nan"), dtype=torch.float64, device="cuda")
    d.work, d.work_bytes = lib.aligned_ptr(buf, 256), int(nb.value)
    f = lib.Functional()
    f.lwt = ctypes.pointer(d)
    rd = torch.tensor(rho, dtype=dt, device="cuda")
    pot = torch.full(nr, float("nan"), dtype=dt, device="cuda")
    en = torch.zeros(lib.NE, dtype=torch.float64, device="cuda")
    lib.check(L.gbofdft_eval(plan.handle, lib.ptr(rd), f, lib.ptr(pot), lib.ptr(en), lib.CALC_E | lib.CALC_V, s))
    torch.cuda.synchronize()

    fr = [2 * np.pi * np.fft.fftfreq(n, d=h) for n in nr]
    q = np.sqrt(fr[0][:, None, None] ** 2 + fr[1][None, :, None] ** 2 + fr[2][None, None, :nr[2] // 2 + 1] ** 2)

    def table(c, end, e):
        j = np.minimum((e / eta[1]).astype(int), neta - 2)
        u = e - eta[j]
        v = c[j, 0] + u * (c[j, 1] + u * (c[j, 2] + u * c[j, 3]))
        return np.where(e < etamax, v, end)

    kmin, kmax = d.kfmin_opt, d.kfmax_opt
    nsp = int(np.ceil(np.log(kmax / kmin) / np.log(ratio))) + 1
    kn = kmin * ratio ** np.arange(nsp)
    assert d.nknots == nsp
    kfc = np.minimum(kf, kmax)
    A = rho ** (5 / 6)
    S = np.fft.rfftn(A)
    inv = lambda z: np.fft.irfftn(z, s=nr, axes=(0, 1, 2))
    pot1, pot3, G, low = np.zeros(nr), np.zeros(nr), np.zeros_like(S), kfc < kn[0]
    for i in range(nsp):
        w = np.zeros(nr)
        if i > 0:
            m = (kfc > kn[i - 1]) & (kfc <= kn[i])
            w[m] = ((kfc - kn[i - 1]) / (kn[i] - kn[i - 1]))[m]
        if i + 1 < nsp:
            m = (kfc > kn[i]) & (kfc <= kn[i + 1])
            w[m] = (1 - (kfc - kn[i]) / (kn[i + 1] - kn[i]))[m]
        K, D = table(kc, fk, q / kn[i]), table(dc, fd, q / kn[i]) / kn[i]
        K[0, 0, 0] = D[0, 0, 0] = 0.0
        pot3 += w * inv(D * S)
        if i == 0:
            w = np.where(low, (kfc - kn[0]) / kn[0], w)
        pot1 += w * inv(K * S)
        G += K * np.fft.rfftn(A * w)
    pot2 = inv(G) if kdd > 1 else pot1
    if kdd < 3:
        pot3[:] = 0.0
    ref = 5 / 6 * A / rho * (pot1 + pot2) + pot3 * kfc / 3 * A / rho
    scale = (A / rho).max() * 4 * max(1.3, 1.0 / kn[0] * kfc.max() / 3) * A.max()
    eps = 2.0 ** -53 if prec else 2.0 ** -24
    tol = (8 * np.log2(N) + 34) * eps
    # a point within rounding of a knot may count to either interval: both give the same sum
    assert np.abs(pot.double().cpu().numpy() - ref).max() <= tol * scale
    assert abs(float(en[lib.E_NL]) - (A * pot1).sum() * dV) <= tol * 2.6 * A.max() * A.sum() * dV
