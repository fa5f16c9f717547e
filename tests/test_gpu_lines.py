"""Line transforms of every kind of length (GPU), each on every axis, against
numpy FP64.

Lengths: one stage (2, 8, 16), FP32 kernels of one length (two stages from 24
to 400 at the smallest, the largest and the radices in between; three stages),
run-time lengths (odd, above 400, seven prime factors), a prime factor above 7
(the run-time-radix passes), a column too long for shared memory.

Tolerance: a transform of n points by stages makes a relative rms error below
eps log2 n (each stage adds at most ~eps); the largest error of a result
stays within 8 eps log2 n of its largest value, eps = 2^-53 or 2^-24.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [2, 8, 16, 24, 36, 42, 56, 81, 84, 90, 96, 100, 105, 128, 144, 150, 160, 162, 192, 196, 216, 250, 256, 288,
           360, 400, 11, 26, 34, 486, 600, 1024]


@pytest.fixture(scope="module")
def lib():
    from dftpy_gb300 import _lib
    _lib.require_cuda()
    return _lib


@pytest.mark.parametrize("prec", [1, 0])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", LENGTHS)
def test_line_lengths(lib, n, axis, prec):
    import torch
    if axis == 2 and n > (600 if prec == 0 else 500):
        pytest.skip("rows longer than a plan takes")
    nr = [5, 6, 4]
    nr[axis] = n
    dt, cdt = (torch.float64, torch.complex128) if prec else (torch.float32, torch.complex64)
    plan = lib.Plan(nr, np.diag([float(k) for k in nr]), precision=prec)      # dV = 1
    rng = np.random.default_rng(n)
    x = rng.standard_normal(nr) + 1.0
    ref = np.fft.rfftn(x)
    tol = 8 * (2.0 ** -53 if prec else 2.0 ** -24) * np.log2(np.prod(nr))
    L = lib.load()
    xd = torch.tensor(x, dtype=dt, device="cuda")
    out = torch.full(ref.shape, float("nan"), dtype=cdt, device="cuda")
    lib.check(L.gbofdft_fft_r2c(plan.handle, lib.ptr(xd), lib.ptr(out), lib.stream_ptr()))
    assert np.abs(out.cpu().numpy() - ref).max() <= tol * np.abs(ref).max()
    sd = torch.tensor(np.ascontiguousarray(ref), dtype=cdt, device="cuda")
    back = torch.full(nr, float("nan"), dtype=dt, device="cuda")
    lib.check(L.gbofdft_fft_c2r(plan.handle, lib.ptr(sd), lib.ptr(back), lib.stream_ptr()))
    assert np.abs(back.cpu().numpy() - x).max() <= tol * np.abs(x).max()
    # forward, table kernel and inverse in one pass of axis 0
    K = np.fft.rfftn(rng.standard_normal(nr)).real
    K = 0.5 * (K + np.fft.rfftn(np.fft.irfftn(K, s=nr, axes=(0, 1, 2))).real)      # an even kernel
    kd = torch.tensor(np.ascontiguousarray(K), dtype=dt, device="cuda")
    conv = torch.full(nr, float("nan"), dtype=dt, device="cuda")
    lib.check(L.gbofdft_convolve(plan.handle, lib.ptr(xd), lib.ptr(conv), lib.KER_ARRAY, lib.ptr(kd), 1.0,
                                 lib.stream_ptr()))
    want = np.fft.irfftn(np.fft.rfftn(x) * K, s=nr, axes=(0, 1, 2))
    assert np.abs(conv.cpu().numpy() - want).max() <= 4 * tol * np.abs(want).max()


@pytest.mark.parametrize("prec", [1, 0])
@pytest.mark.parametrize("nr", [(12, 10, 14), (9, 15, 7), (22, 6, 8), (8, 7, 5)])
def test_c2r_input_alignment(lib, nr, prec):
    """The first inverse pass reads the caller's spectrum where it is aligned to a
    complex value (else a copy of it): the same values, and the input is left alone."""
    import torch
    dt = torch.float64 if prec else torch.float32
    plan = lib.Plan(nr, np.diag([float(k) for k in nr]), precision=prec)
    L = lib.load()
    X = np.fft.rfftn(np.random.default_rng(3).standard_normal(nr))
    flat = torch.tensor(np.ascontiguousarray(X).view(np.float64).reshape(-1), dtype=dt, device="cuda")
    res = []
    for off in (0, 1, 2):
        buf = torch.zeros(flat.numel() + 4, dtype=dt, device="cuda")
        buf[off:off + flat.numel()] = flat
        keep = buf.clone()
        out = torch.full(nr, float("nan"), dtype=dt, device="cuda")
        p = buf.data_ptr() + off * buf.element_size()
        lib.check(L.gbofdft_fft_c2r(plan.handle, p, lib.ptr(out), lib.stream_ptr()))
        assert torch.equal(buf, keep)
        res.append(out)
    assert torch.equal(res[0], res[1]) and torch.equal(res[0], res[2])
    want = np.fft.irfftn(X, s=nr, axes=(0, 1, 2))
    tol = 8 * (2.0 ** -53 if prec else 2.0 ** -24) * np.log2(np.prod(nr))
    assert np.abs(res[0].cpu().numpy() - want).max() <= tol * np.abs(want).max()
