"""Every length that has line kernels of its own (GPU), on every axis: forward,
inverse and convolution against numpy FP64, FP32 plans.

Tolerance: a transform of N points by stages makes a relative rms error below
eps log2 N; the largest error of a result stays within 8 eps log2 N of its
largest value, eps = 2^-24."""
import os
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
with open(os.path.join(os.path.dirname(HERE), "dftpy_gb300", "csrc", "passes_rb.cuh")) as _f:
    LENGTHS = sorted(int(n) for n in re.findall(r"X\((\d+), GB_RB_G", _f.read()))


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", LENGTHS)
def test_compiled_length(n, axis):
    import torch
    from dftpy_gb300 import _lib as lib
    lib.require_cuda()
    nr = [5, 4, 6]
    nr[axis] = n
    plan = lib.Plan(nr, np.diag([float(k) for k in nr]), precision=0)      # dV = 1
    L, s = lib.load(), lib.stream_ptr()
    rng = np.random.default_rng(n)
    x = rng.standard_normal(nr) + 1.0
    X = np.fft.rfftn(x)
    tol = 8 * 2.0 ** -24 * np.log2(np.prod(nr))
    xd = torch.tensor(x, dtype=torch.float32, device="cuda")
    out = torch.full(X.shape, float("nan"), dtype=torch.complex64, device="cuda")
    lib.check(L.gbofdft_fft_r2c(plan.handle, lib.ptr(xd), lib.ptr(out), s))
    assert np.abs(out.cpu().numpy() - X).max() <= tol * np.abs(X).max()
    sd = torch.tensor(np.ascontiguousarray(X), dtype=torch.complex64, device="cuda")
    back = torch.full(nr, float("nan"), dtype=torch.float32, device="cuda")
    lib.check(L.gbofdft_fft_c2r(plan.handle, lib.ptr(sd), lib.ptr(back), s))
    assert np.abs(back.cpu().numpy() - x).max() <= tol * np.abs(x).max()
    conv = torch.full(nr, float("nan"), dtype=torch.float32, device="cuda")
    lib.check(L.gbofdft_convolve(plan.handle, lib.ptr(xd), lib.ptr(conv), lib.KER_NONE, None, 1.0, s))
    assert np.abs(conv.cpu().numpy() - x).max() <= 4 * tol * np.abs(x).max()
