"""Pointwise terms of the evaluation's row passes (GPU): densities that the
clamps meet, against the clamps written out in numpy."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KZ = 1e-30
# rows of kernels of one length, of run-time lengths (odd, above 400), of a prime factor above 7
LENGTHS = [36, 128, 105, 486, 22]


@pytest.fixture(scope="module")
def lib():
    from dftpy_gb300 import _lib
    _lib.require_cuda()
    return _lib


def _plan(lib, nr, prec):
    return lib.Plan(nr, np.diag([0.4 * k for k in nr]), precision=prec)


def _eval(lib, plan, f, rho, energies=True):
    """Potential and energies of the functional ``f`` at ``rho`` (numpy)."""
    import torch
    r = torch.tensor(rho, dtype=torch.float64 if plan.precision == lib.F64 else torch.float32, device="cuda")
    pot = torch.full_like(r, 7.0)
    en = torch.zeros(lib.NE, dtype=torch.float64, device="cuda")
    lib.check(lib.load().gbofdft_eval(plan.handle, lib.ptr(r), ctypes.byref(f), lib.ptr(pot), lib.ptr(en),
                                      lib.CALC_V | (lib.CALC_E if energies else 0), lib.stream_ptr()))
    torch.cuda.synchronize()
    return pot.cpu().numpy(), en.cpu().numpy()


@pytest.mark.parametrize("prec", [1, 0])
@pytest.mark.parametrize("beta", [5 / 6, 0.7])
@pytest.mark.parametrize("n2", LENGTHS)
def test_nan_density_reaches_the_power(lib, n2, beta, prec):
    """A NaN of the density is one of rho^beta, and the convolution carries it to every
    point of the Wang-Teter potential: a broken density must not look like a good one."""
    import torch
    nr = (6, 5, n2)
    plan = _plan(lib, nr, prec)
    kern = torch.ones((6, 5, n2 // 2 + 1), dtype=torch.float64 if prec else torch.float32, device="cuda")
    f = lib.Functional()
    f.wt, f.wt_alpha, f.wt_beta, f.wt_kernel = 1, beta, beta, kern.data_ptr()
    rho = np.full(nr, 0.03)
    assert np.isfinite(_eval(lib, plan, f, rho)[0]).all()
    rho[3, 2, n2 // 3] = np.nan
    pot, en = _eval(lib, plan, f, rho)
    assert np.isnan(pot).all() and np.isnan(en[lib.E_NL])


@pytest.mark.parametrize("prec", [1, 0])
@pytest.mark.parametrize("rows", [(2, 3), (1, 1), (12, 10)])
@pytest.mark.parametrize("n2", LENGTHS[:4] + [84, 400, 8])
def test_energy_sums(lib, n2, rows, prec):
    """Energies that are sums of products of two fields of the plan's precision.

    Tolerance: the products are exact to twice the precision and a thread's n <= 64
    points add an error below n^2 2^-49 = 8e-12 of the magnitudes' sum (FP32), n 2^-53
    (FP64); the additions above are FP64, below 64 2^-53."""
    import math
    import torch
    nr = rows + (n2,)
    plan = _plan(lib, nr, prec)
    dt = np.float64 if prec else np.float32
    rng = np.random.default_rng(n2)
    rho = (0.03 + 0.02 * rng.random(nr)).astype(dt)
    vloc = (1.0 + rng.random(nr)).astype(dt)
    dV = 0.4 ** 3
    tol = 128 * 2.0 ** -53 if prec else 1e-11
    vd = torch.tensor(vloc, device="cuda")
    f = lib.Functional()
    f.vloc = vd.data_ptr()
    pot, en = _eval(lib, plan, f, rho)
    assert np.array_equal(pot, vloc)
    terms = (rho.astype(float) * vloc.astype(float)).ravel()       # exact in FP32's case
    want = math.fsum(terms) * dV
    assert abs(en[lib.E_PSEUDO] - want) <= tol * want
    f = lib.Functional()
    f.hartree = 1
    pot, en = _eval(lib, plan, f, rho)
    terms = (0.5 * rho.astype(float) * pot.astype(float)).ravel()
    assert abs(en[lib.E_HARTREE] - math.fsum(terms) * dV) <= tol * np.abs(terms).sum() * dV


@pytest.mark.parametrize("prec", [1, 0])
@pytest.mark.parametrize("n2", [36, 84, 128, 105])
def test_pointwise_rounding(lib, n2, prec):
    """Thomas-Fermi and LDA potentials to the roundings that their operations make.

    One rounding is off by at most u = 2^-53 or 2^-24 of its value, 0.45 u rms.  x^(-1/3)
    and x^(1/3) come out of a correction by a residual with one or two roundings, a third
    of which reaches them: 0.5 u rms.  Thomas-Fermi is two products further (0.8 u rms);
    LDA's exchange one product and one sum further, its correlation, below a fifth of it
    here, a dozen operations long (1.2 u)."""
    nr = (24, 20, n2)
    plan = _plan(lib, nr, prec)
    dt = np.float64 if prec else np.float32
    u = 2.0 ** -53 if prec else 2.0 ** -24
    rho = np.exp(np.random.default_rng(n2).uniform(np.log(3e-3), np.log(0.3), nr)).astype(dt)
    one = np.longdouble(1)
    x = rho.astype(np.longdouble)
    c = x ** (one / 3)
    k = lambda v: np.longdouble(dt(v))                  # the constants as the device has them
    f = lib.Functional()
    f.tf, f.tf_x = 1, 1.0
    pot, _ = _eval(lib, plan, f, rho, energies=False)
    want = np.longdouble(4.78539000031365302657) * c * c
    err = ((pot - want) / want).astype(float) / u
    assert np.sqrt((err * err).mean()) <= 1.0
    f = lib.Functional()
    f.xc = 1
    pot, _ = _eval(lib, plan, f, rho, energies=False)
    a, b, cc, d, g, b1, b2 = (k(v) for v in (0.0311, -0.048, 0.0020, -0.0116, -0.1423, 1.0529, 0.3334))
    rs = k(0.62035049089940001667) / c
    lr, sq = np.log(rs), np.sqrt(rs)
    vc = np.where(rs < 1, lr * (a + 2 * one / 3 * cc * rs) + b - a / 3 + (2 * d - cc) * rs / 3,
                  (g + 7 * one / 6 * g * b1 * sq + 4 * one / 3 * g * b2 * rs) / (1 + b1 * sq + b2 * rs) ** 2)
    want = vc - k(0.98474502184269654115) * c
    err = ((pot - want) / want).astype(float) / u
    assert np.sqrt((err * err).mean()) <= 1.2
