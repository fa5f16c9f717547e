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


@pytest.mark.parametrize("prec", [1, 0])
@pytest.mark.parametrize("beta", [5 / 6, 0.7])
@pytest.mark.parametrize("n2", LENGTHS)
def test_densities_that_are_clamped(lib, n2, beta, prec):
    """Zero, negative and tiny densities: the terms written out with their clamps.

    Tolerance: a convolution with kernel K of a field x errs below 16 eps log2 N max|K|
    rms(x); the factors around it and the local terms make a dozen roundings, their
    products with the convolution included (32 eps of the value).  rho^2 under
    Thomas-Fermi's cube root loses what lies below the smallest normal FP32 number, and
    LDA's correlation, 0.19 / den, is lost where den^2 is above the largest one."""
    import torch
    nr = (6, 4, n2)
    plan = _plan(lib, nr, prec)
    dt = np.float64 if prec else np.float32
    eps = 2.0 ** -53 if prec else 2.0 ** -24
    rng = np.random.default_rng(n2)
    rho = (0.03 + 0.02 * rng.random(nr)).astype(dt)
    odd = np.array([0.0, -0.0, -1e-3, -1e-31, 1e-31, 5e-31, 1e-30, 2e-30, 1e-24, 1e-12, 1e-7], dtype=dt)
    where = rng.choice(rho.size, 3 * odd.size, replace=False)
    rho.reshape(-1)[where] = np.tile(odd, 3)
    r = rho.astype(float)
    kz = float(dt(KZ))
    N, dV = rho.size, 0.4 ** 3
    log2n = np.log2(N)
    m = np.meshgrid(*[np.fft.fftfreq(n, 1.0 / n) for n in nr[:2]], np.arange(n2 // 2 + 1), indexing="ij")
    gg = sum((2 * np.pi * mi / (0.4 * n)) ** 2 for mi, n in zip(m, nr))

    def conv(K, x):
        return (np.fft.irfftn(K * np.fft.rfftn(x), s=nr, axes=(0, 1, 2)),
                16 * eps * log2n * np.abs(K).max() * np.sqrt((x * x).mean()))

    def check(f, slot, pot, terms, err):
        """err: the potential's error at each point, beside 32 eps of its value."""
        got, en = _eval(lib, plan, f, rho)
        bound = err + 32 * eps * np.abs(pot) + 1e-37
        assert (np.abs(got - pot) <= bound).all()
        assert abs(en[slot] - terms.sum() * dV) <= 2 * (np.abs(r) * bound + 32 * eps * np.abs(terms)).sum() * dV

    f = lib.Functional()
    f.tf, f.tf_x = 1, 1.0
    c = np.cbrt(r)
    check(f, lib.E_TF, 4.78539000031365302657 * c * c, 2.87123400018819181594 * c ** 5,
          np.full(nr, 0.0 if prec else 5.0 * np.cbrt(2.0 ** -126)))
    f = lib.Functional()
    f.vw, f.vw_y = 1, 1.0
    rm = np.where(r > 0, r, kz)
    sq = np.sqrt(rm)
    w, e = conv(gg, sq)
    v = 0.5 * w / sq
    check(f, lib.E_VW, v, np.where(r > 0, r * v, 0.0), 0.5 * e / sq)
    f = lib.Functional()
    K = 1.0 / (1.0 + gg)
    kd = torch.tensor(K.astype(dt), device="cuda")
    f.wt, f.wt_alpha, f.wt_beta, f.wt_kernel = 1, beta, beta, kd.data_ptr()
    rc = np.where(r < kz, kz, r)
    kc, e = conv(K.astype(dt).astype(float), rc ** beta)
    v = 2 * beta * rc ** (beta - 1) * kc
    # rc^(beta - 1): the exponent's rounding is one of |ln rc| roundings
    check(f, lib.E_NL, v, v * r / (2 * beta), 2 * beta * rc ** (beta - 1) * e + 70 * eps * np.abs(v))
    f = lib.Functional()
    f.xc = 1
    c = np.maximum(np.cbrt(r), kz)
    rs = 0.62035049089940001667 / c
    sq, lr = np.sqrt(rs), np.log(rs)
    den = 1 + 1.0529 * sq + 0.3334 * rs
    cx = 0.98474502184269654115
    low = rs >= 1
    vx = -cx * c + np.where(low, (-0.1423 - 0.1423 * (7 / 6 * 1.0529 * sq + 4 / 3 * 0.3334 * rs)) / den ** 2,
                            lr * (0.0311 + 2 / 3 * 0.002 * rs) - 0.048 - 0.0311 / 3 + (2 * -0.0116 - 0.002) * rs / 3)
    ex = -0.75 * cx * c + np.where(low, -0.1423 / den, 0.0311 * lr - 0.048 + 0.002 * rs * lr - 0.0116 * rs)
    check(f, lib.E_XC, vx, ex * r, np.full(nr, 0.0 if prec else 0.19 * 2.0 ** -63))


@pytest.mark.parametrize("power", [-70, -40, 40, 70])
def test_hartree_of_any_cell_size(lib, power):
    """The Hartree potential of a cell scaled by s is s^2 times the cell's, also where
    |G|^2 and its reciprocal leave the FP32 range."""
    nr = (12, 10, 14)
    rho = 0.03 + 0.02 * np.random.default_rng(1).random(nr)
    f = lib.Functional()
    f.hartree = 1
    s = 2.0 ** power
    want = _eval(lib, _plan(lib, nr, 1), f, rho, energies=False)[0] * s * s
    plan = lib.Plan(nr, np.diag([0.4 * s * k for k in nr]), precision=1)
    got = _eval(lib, plan, f, rho, energies=False)[0]
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()
