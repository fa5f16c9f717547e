"""Ewald real-space pairs (GPU): the single-precision test that leaves far pairs
out drops none within the cutoff -- ions far from the origin, pairs at the
cutoff to a few parts in 1e7, fewer ions than threads and more -- and the
spline interval found from a single-precision guess is the bisection's.

Tolerances: the terms are positive, erfc and the root good to a few eps: the sums
agree to 64 eps.  The potential of one ion is the spline itself: 1e-13.
"""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0.0, 37.0, 4000.0])
@pytest.mark.parametrize("nat", [1, 7, 300])
def test_real_space_sum(nat, shift):
    import torch
    from dftpy_gb300 import _lib as lib
    lib.require_cuda()
    L = lib.load()
    lat = np.diag([11.0, 12.0, 13.0])
    rng = np.random.default_rng(nat)
    pos = rng.random((nat, 3)) @ lat + shift
    rmax, eta = 7.3, 0.2
    if nat > 2:                                   # pairs on either side of the cutoff
        pos[1] = pos[0] + [rmax * (1 - 3e-7), 0, 0]
        pos[2] = pos[0] + [0, rmax * (1 + 3e-7), 0]
    q = rng.uniform(1.0, 3.0, nat)
    rg = np.arange(-1, 2)
    img = np.array(np.meshgrid(rg, rg, rg, indexing="ij")).reshape(3, -1).T.astype(float) @ lat
    plan = lib.Plan((8, 8, 8), lat, precision=1)
    nb = lib.setup_workspace_bytes(plan, nat)
    work = torch.empty(nb // 8 + 64, dtype=torch.float64, device="cuda")
    dev = [torch.tensor(np.ascontiguousarray(a), device="cuda") for a in (pos, (pos @ np.linalg.inv(lat)) % 1.0, q, img)]
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    lib.check(L.gbofdft_ewald(plan.handle, nat, lib.ptr(dev[0]), lib.ptr(dev[1]), lib.ptr(dev[2]), eta, rmax,
                              lib.ptr(dev[3]), len(img), 0, 10, None, lib.aligned_ptr(work, 256), nb, lib.ptr(out),
                              lib.stream_ptr()))
    want = 0.0
    erfc = np.vectorize(math.erfc, otypes=[float])
    for i in range(nat):
        r = pos[i] - (pos[None, :, :] - img[:, None, :])
        d = np.sqrt((r * r).sum(-1))
        m = (d < rmax) & (d > 0.001)
        qq = np.broadcast_to(q, d.shape)[m]
        want += 0.5 * q[i] * (qq * erfc(math.sqrt(eta) * d[m]) / d[m]).sum()
    # coordinates near 4000 carry the distances to 1e-12 only, on both sides alike but for rounding
    tol = 64 * 2.0 ** -53 * (1.0 + shift)
    assert abs(float(out[0]) - want) <= tol * max(want, 1e-3) * 8


@pytest.mark.parametrize("kind", ["uniform", "log", "jitter"])
@pytest.mark.parametrize("m", [4, 5, 1000, 20000])
def test_spline_interval(m, kind):
    import torch
    from dftpy_gb300 import _lib as lib
    from dftpy_gb300._tables import spline_notaknot
    lib.require_cuda()
    rng = np.random.default_rng(m)
    x = np.linspace(0.5, 9.0, m)
    if kind == "log":
        x = np.geomspace(0.5, 9.0, m)
    elif kind == "jitter":
        x = x + rng.uniform(-0.4, 0.4, m) * (x[1] - x[0])
    y = np.cos(x)
    _, c = spline_notaknot(x, y)
    lat = np.diag([8.0, 9.0, 10.0])
    nr = (12, 10, 14)
    plan = lib.Plan(nr, lat, precision=1)
    xd, cd = (torch.tensor(np.ascontiguousarray(a).reshape(-1), device="cuda") for a in (x, c))
    t = (lib.VTable * 1)()
    t[0].x, t[0].c, t[0].m = xd.data_ptr(), cd.data_ptr(), m
    for i in range(5):
        t[0].q4[i] = 0.0
    t[0].dp, t[0].gmin, t[0].gmax = 1.0, float(x[0]), float(x[-1])
    nb = lib.setup_workspace_bytes(plan, 1)
    work = torch.empty(nb // 8 + 64, dtype=torch.float64, device="cuda")
    spos = torch.zeros((1, 3), dtype=torch.float64, device="cuda")      # at the origin: v(G) = vline(|G|)
    sp = torch.zeros(1, dtype=torch.int32, device="cuda")
    v = torch.empty((12, 10, 8), dtype=torch.complex128, device="cuda")
    lib.check(lib.load().gbofdft_vloc(plan.handle, 1, t, 1, lib.ptr(spos), lib.ptr(sp), 0, 10, None,
                                      lib.aligned_ptr(work, 256), nb, lib.ptr(v), None, lib.stream_ptr()))
    f = [2 * np.pi * np.fft.fftfreq(n, d=l / n) for n, l in zip(nr, np.diag(lat))]
    q = np.sqrt(f[0][:, None, None] ** 2 + f[1][None, :, None] ** 2 + (np.arange(8) * 2 * np.pi / 10.0)[None, None, :] ** 2)
    j = np.clip(np.searchsorted(x, q, side="right") - 1, 0, m - 2)
    u = q - x[j]
    want = np.where((q >= x[0]) & (q < x[-1]), c[j, 0] + u * (c[j, 1] + u * (c[j, 2] + u * c[j, 3])), 0.0)
    got = v.cpu().numpy()
    scale = np.abs(c).max(axis=0) @ np.array([1.0, *(np.diff(x).max() ** np.arange(1, 4))])
    edge = (np.abs(q - x[0]) < 1e-12) | (np.abs(q - x[-1]) < 1e-12)
    assert np.abs((got - want)[~edge]).max() <= 1e-13 * scale
