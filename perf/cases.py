"""Performance cases: the work a program using this package has it do.

Every case goes through the public classes (``DirectGrid``, ``DirectField``,
``TotalFunctional``, ``LocalPseudo``, ``Optimization``).  Kinds:

``eval``   one ``TotalFunctional`` evaluation -- the inner loop of every density
           optimisation.  FP64 calls ask for energy and potential (what a line
           search asks for), FP32 calls for the potential alone (what the
           Hessian products of a truncated-Newton step ask for).
``fft``    ``DirectField.fft()``, a reciprocal-space filter and ``ifft()``: a
           program's own reciprocal-space work on a field.
``ions``   one step of a relaxation or of molecular dynamics at a given
           density: new positions, local pseudopotential, ion-ion energy, forces.
``solve``  one whole mixed-precision density optimisation.

Grids are the workloads' own (32^3, 96^3 ... 160^3, 360^3) and the other sizes
that ``DirectGrid(lattice, spacing=...)`` picks (even, 2, 3, 5, 7-smooth) or
that a density file brings (odd ones too); cells are fcc Al and Al/Mg at 0.2 to
0.4 Bohr spacing, orthorhombic or skewed, on half and full reciprocal grids.
"""
import math

import numpy as np
import torch

from dftpy_gb300 import functional as F
from dftpy_gb300 import systems
from dftpy_gb300.batch import build_evaluator
from dftpy_gb300.field import DirectField, ReciprocalField
from dftpy_gb300.grid import DirectGrid
from dftpy_gb300.ions import Ions
from dftpy_gb300.optimization import Optimization

A0 = 7.65                     # fcc lattice constant (Bohr)
PI = math.pi
C_TF = 0.3 * (3.0 * PI ** 2) ** (2.0 / 3.0)


def _case(name, kind, kedf, nr, reps, dtype, full=False, skew=False, mg=0.0):
    c = {"kind": kind, "kedf": kedf, "n0": nr[0], "n1": nr[1], "n2": nr[2], "r0": reps[0], "r1": reps[1],
         "r2": reps[2], "dtype": dtype, "full": full, "skew": skew, "mg": mg}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the 4-atom cell: launch and call latency
        _case("eval_tfvw_fp64_32", "eval", "TFVW", (32, 32, 32), (1, 1, 1), "fp64"),
        # the 256-atom cell with the Wang-Teter functional: line-search and Hessian evaluations
        _case("eval_wt_fp64_128", "eval", "WT", (128, 128, 128), (4, 4, 4), "fp64"),
        _case("eval_wt_fp32_128", "eval", "WT", (128, 128, 128), (4, 4, 4), "fp32"),
        # alloy snapshots with the density-dependent kernel, smallest grid in FP64, an orthorhombic one in FP32
        _case("eval_wgc_fp64_96", "eval", "WGC", (96, 96, 96), (3, 3, 3), "fp64", mg=0.15),
        _case("eval_wgc_fp32_96x128x160", "eval", "WGC", (96, 128, 160), (3, 4, 5), "fp32", mg=0.15),
        # grids picked from a spacing: the default full reciprocal grid and a skewed cell; an orthorhombic alloy
        _case("eval_wt_fp64_84x90x100", "eval", "WT", (84, 90, 100), (3, 3, 3), "fp64", full=True, skew=True),
        _case("eval_wgc_fp32_108x120x144", "eval", "WGC", (108, 120, 144), (3, 4, 5), "fp32", mg=0.15),
        # the density-dependent LMGP functional: a small cell in FP64 and the 4000-atom one in FP32
        _case("eval_lmgp_fp64_64x64x80", "eval", "LMGP", (64, 64, 80), (2, 2, 3), "fp64"),
        _case("eval_lmgp_fp32_360", "eval", "LMGP", (360, 360, 360), (10, 10, 10), "fp32"),
        # a program's own filter of a field
        _case("fft_fp64_180x192x200", "fft", "", (180, 192, 200), (6, 6, 6), "fp64"),
        # a relaxation step of the largest alloy snapshot
        _case("ions_fp64_160", "ions", "WGC", (160, 160, 160), (5, 5, 5), "fp64", mg=0.15),
        # a whole optimisation of the smallest alloy snapshot
        _case("solve_mixed_96", "solve", "WGC", (96, 96, 96), (3, 3, 3), "mixed", mg=0.15),
    ]


def _smooth(n, primes):
    for p in primes:
        while n % p == 0:
            n //= p
    return n == 1


EVEN = [n for n in range(16, 361, 2) if _smooth(n, (2, 3, 5, 7))]
ODD = [n for n in range(15, 160, 2) if _smooth(n, (3, 5, 7, 11, 13, 17))]


def draw(rng):
    kind = rng.choices(["eval", "fft", "ions", "solve"], [0.7, 0.12, 0.1, 0.08])[0]
    if kind == "solve":
        # the alloy snapshots' own grids, and grids of the same cells picked from other spacings
        return _case("", "solve", "WGC", *rng.choice([((96, 96, 96), (3, 3, 3)), ((96, 96, 128), (3, 3, 4)),
                                                     ((96, 128, 128), (3, 4, 4)), ((96, 128, 160), (3, 4, 5)),
                                                     ((84, 84, 84), (3, 3, 3)), ((90, 108, 120), (3, 4, 4))]),
                     "mixed", mg=rng.choice([0.05, 0.1, 0.2, 0.25]))
    dtype = rng.choice(["fp64", "fp32"]) if kind != "ions" else "fp64"
    kedf = rng.choice(["TFVW", "WT", "WT", "WGC", "WGC", "LMGP"]) if kind == "eval" else ("" if kind == "fft" else "WT")
    top = {"TFVW": 240, "WT": 240, "WGC": 180, "LMGP": 128, "": 240}[kedf]
    if dtype == "fp64" and kind != "fft":
        top = min(top, 160)
    while True:
        side = 24.0 * (top / 24.0) ** rng.random()            # sizes evenly over their logarithm
        pick = ODD if rng.random() < 0.15 else EVEN
        nr = []
        for _ in range(3):
            want = side * rng.uniform(0.75, 1.33)
            nr.append(min(pick, key=lambda n: abs(n - want)))
        if max(nr) <= 360 and nr[0] * nr[1] * nr[2] <= top ** 3:
            break
    h = rng.uniform(0.2, 0.36)
    reps = [max(1, round(n * h / A0)) for n in nr]
    full = rng.random() < 0.4
    return _case("", kind, kedf, nr, reps, dtype, full=full, skew=rng.random() < 0.3,
                 mg=0.15 if kedf in ("WGC", "LMGP") else 0.0)


# ---- inputs ----------------------------------------------------------------
def _structure(c, seed):
    """fcc Al or Al/Mg with jittered positions; skewed cells shear the same fractional coordinates."""
    st = systems.fcc_supercell((c["r0"], c["r1"], c["r2"]), a=A0, sigma=0.1, seed=int(seed) % (1 << 31),
                               nr=(c["n0"], c["n1"], c["n2"]), mg_fraction=c["mg"])
    if c["skew"]:
        shear = np.array([[1.0, 0.0, 0.0], [0.12, 1.0, 0.0], [-0.07, 0.09, 1.0]])
        st.positions = st.positions @ np.linalg.inv(st.lattice) @ (st.lattice @ shear)
        st.lattice = st.lattice @ shear
    return st


def _density(c, seed, st):
    """A density like a converged one on the GPU (FP64): maxima at the fcc sites of ~8 times the mean, random long
    waves, normalised to the valence electrons."""
    r = np.random.default_rng(int(seed) % (1 << 31) + 77)
    nr, reps = (c["n0"], c["n1"], c["n2"]), (c["r0"], c["r1"], c["r2"])
    s = [torch.arange(n, device="cuda", dtype=torch.float64) / n for n in nr]
    waves = [(0.35, (1, 1, 1), 0.0), (0.35, (-1, 1, 1), 0.0), (0.35, (1, -1, 1), 0.0), (0.35, (1, 1, -1), 0.0),
             (0.2, (2, 0, 0), 0.0), (0.2, (0, 2, 0), 0.0), (0.2, (0, 0, 2), 0.0)]
    waves = [(a * r.uniform(0.9, 1.1), tuple(m * k for m, k in zip(w, reps)), p) for a, w, p in waves]
    waves += [(r.uniform(0.03, 0.12), tuple(int(x) for x in r.integers(-2, 3, 3)), r.uniform(0, 2 * PI))
              for _ in range(6)]
    # a separable sum: Re of outer products of the axes' phases
    amp = torch.tensor([a for a, _, _ in waves], device="cuda", dtype=torch.float64)
    ph = [torch.polar(torch.ones(len(waves), n, device="cuda", dtype=torch.float64),
                      torch.stack([2 * PI * w[d] * s[d] for _, w, _ in waves])) for d, n in enumerate(nr)]
    p0 = torch.polar(amp, torch.tensor([p for _, _, p in waves], device="cuda", dtype=torch.float64))
    left = (p0[:, None, None] * ph[0][:, :, None] * ph[1][:, None, :]).reshape(len(waves), -1)
    x = (left.real.T @ ph[2].real - left.imag.T @ ph[2].imag).reshape(nr)
    x = torch.exp(x)
    return x * (st.nelec / st.volume / x.mean())


def _ions(st):
    return Ions(st.symbols, positions=st.positions, cell=st.lattice)


def _evaluator(c, st, grid):
    pp = {s: F.AnalyticPP(*systems.SPECIES[s]) for s in set(st.symbols)}
    ps = F.LocalPseudo(grid=grid, ions=_ions(st), PP_list=pp, PME=True)
    return F.TotalFunctional(KineticEnergyFunctional=F.Functional(type="KEDF", name=c["kedf"]),
                             XCFunctional=F.Functional(type="XC", name="LDA"),
                             HARTREE=F.Functional(type="HARTREE"), PSEUDO=ps)


def prepare(case, seed):
    c = case
    st = _structure(c, seed)
    if c["kind"] == "solve":
        total, rho0 = build_evaluator(st, kedf=c["kedf"])
        return {"kind": "solve", "total": total, "rho": rho0, "nat": st.nat}
    grid = DirectGrid(st.lattice, st.nr, full=c["full"])
    dtype = torch.float64 if c["dtype"] == "fp64" else torch.float32
    rho = DirectField(grid, data=_density(c, seed, st).to(dtype))
    state = {"kind": c["kind"], "rho": rho, "grid": grid}
    if c["kind"] == "fft":
        # a Gaussian filter on the reciprocal grid, as a program that smooths a field keeps it
        rg = grid.get_reciprocal()
        state["recip"] = rg
        state["filter"] = torch.exp(-0.05 * rg.gg).to(dtype)
        return state
    state["total"] = _evaluator(c, st, grid)
    if c["kind"] == "ions":
        state["ions"] = _ions(st)
    else:
        state["calc"] = {"E", "V"} if c["dtype"] == "fp64" else {"V"}
    return state


# ---- one pass --------------------------------------------------------------
def run(state):
    kind = state["kind"]
    rho = state["rho"]
    if kind == "eval":
        out = state["total"].compute(rho, calcType=state["calc"])
        v = out.potential.as_subclass(torch.Tensor)
        return {"energy": out.energy, "potential": v} if "E" in state["calc"] else {"potential": v}
    if kind == "fft":
        g = rho.fft()
        g = ReciprocalField(state["recip"], data=g.as_subclass(torch.Tensor) * state["filter"])
        return {"spectrum": g.as_subclass(torch.Tensor), "field": g.ifft().as_subclass(torch.Tensor)}
    if kind == "ions":
        total = state["total"]
        total.PSEUDO.restart(ions=state["ions"], grid=state["grid"])
        v = total.PSEUDO.vreal.as_subclass(torch.Tensor)
        e = float(total.ewald.energy)
        return {"v_loc": v, "e_ion": e, "forces": total.get_forces(rho)}
    opt = Optimization(EnergyEvaluator=state["total"], optimization_method="TN",
                       optimization_options={"econv": 1e-8 * state["nat"], "maxfun": 50, "maxiter": 100,
                                             "precision": "mixed"})
    r = opt.optimize_rho(guess_rho=state["rho"])
    # the training sets of the density-guess network keep sqrt(rho) in single precision
    return {"energy": opt.energy, "sqrt_rho": torch.sqrt(torch.clamp(r.as_subclass(torch.Tensor).to(torch.float32),
                                                                     min=1e-12))}


# ---- what a pass cannot do without -----------------------------------------
TRANSFORMS = {"TFVW": 4, "WT": 6, "WGC": 16}


def work(case):
    c = case
    n = c["n0"] * c["n1"] * c["n2"]
    s = 8 if c["dtype"] == "fp64" else 4
    ng = c["n0"] * c["n1"] * (c["n2"] // 2 + 1)
    one = 2.5 * n * math.log2(n)                       # a real transform
    nat = 4 * c["r0"] * c["r1"] * c["r2"]
    if c["kind"] == "eval":
        tables = {"TFVW": 0, "WT": 1, "WGC": 4, "LMGP": 0}[c["kedf"]]
        nt = 4 + 3 * 14 if c["kedf"] == "LMGP" else TRANSFORMS[c["kedf"]]     # LMGP: ~14 knots in these densities
        return {"bytes": s * (3 * n + tables * ng), "flops": nt * one + 100.0 * n}
    if c["kind"] == "fft":
        k = n if c["full"] else ng
        return {"bytes": s * (2 * n + 2 * k + k), "flops": 2 * one + 2.0 * k}
    if c["kind"] == "ions":
        # v_loc and the PME sums: transforms of the species' and the total charge, of v_loc and of two force fields
        nt = 5 + (1 if c["mg"] > 0 else 0)
        return {"bytes": s * 2 * n, "flops": nt * one + nat * 1000.0 * 20}
    # solve: about 25 FP32 and a few FP64-accurate evaluations of 16 transforms
    return {"bytes": 30 * 4 * (3 * n + 4 * ng), "flops": 30 * (16 * one + 100.0 * n)}


# ---- the values in 64 bits, by plain tensor algebra --------------------------
class _Box:
    """Reciprocal geometry and transforms in FP64, in the convention of full or half reciprocal grids."""

    def __init__(self, c, lattice):
        self.n = (c["n0"], c["n1"], c["n2"])
        self.full = c["full"]
        self.vol = abs(float(np.linalg.det(lattice)))
        self.N = self.n[0] * self.n[1] * self.n[2]
        self.dV = self.vol / self.N
        b = 2 * PI * np.linalg.inv(lattice).T
        ax = [torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda") for n in self.n]
        if not self.full:
            ax[2] = torch.arange(self.n[2] // 2 + 1, dtype=torch.float64, device="cuda")
        self.m = ax
        m = torch.meshgrid(*ax, indexing="ij")
        self.gg = sum(sum(float(b[j, k]) * m[j] for j in range(3)) ** 2 for k in range(3))
        self.b = b

    def fwd(self, x):
        return torch.fft.fftn(x) if self.full else torch.fft.rfftn(x)

    def inv(self, X):
        if self.full:
            return torch.fft.ifftn(X).real.contiguous()
        X = torch.fft.ifftn(X, dim=(0, 1))
        edge = X.clone()
        for k in {0} | ({self.n[2] // 2} if self.n[2] % 2 == 0 else set()):
            edge[:, :, k] = X[:, :, k].real.to(X.dtype)
        return torch.fft.irfft(edge, n=self.n[2], dim=2)

    def conv(self, x, K):
        return self.inv(self.fwd(x) * K)

    def phases(self, scaled):
        """exp(-2 pi i m_d s_d) per atom and axis."""
        s = torch.tensor(scaled, dtype=torch.float64, device="cuda")
        return [torch.polar(torch.ones((), dtype=torch.float64, device="cuda").expand(len(s), len(self.m[d])),
                            -2 * PI * torch.remainder(s[:, d:d + 1] * self.m[d][None, :], 1.0)) for d in range(3)]

    def structure(self, ph, w):
        """sum_a w_a exp(-i G.R_a) on the grid."""
        left = (ph[0] * w[:, None])[:, :, None] * ph[1][:, None, :]
        return (left.reshape(len(w), -1).T @ ph[2]).reshape(len(self.m[0]), len(self.m[1]), len(self.m[2]))


def _inverse_lindhard(eta):
    """1/F - 3 eta^2 - 1 with F = 1/2 + (1 - eta^2)/(4 eta) ln|(1 + eta)/(1 - eta)| = sum_k eta^-2k / (4 k^2 - 1)."""
    eta = torch.as_tensor(eta, dtype=torch.float64)
    e = torch.clamp(eta, 1e-8, None)
    small = torch.clamp(e, None, 3.0)
    d = torch.clamp(torch.abs(1 - small), 1e-300)
    f = 0.5 + (1 - small ** 2) / (4 * small) * torch.log((1 + small) / d)
    lo = 1 / f - 3 * small ** 2 - 1
    y = 1 / torch.clamp(e, 3.0, None) ** 2
    # F = y/3 (1 + r): 1/F - 3/y = -(3/y) r / (1 + r), r = y sum_{k>=2} 3 y^(k-2) / (4 k^2 - 1)
    r = torch.zeros_like(y)
    for k in range(40, 1, -1):
        r = r * y + 3.0 / (4 * k * k - 1)
    hi = -3 * r / (1 + r * y) - 1
    out = torch.where(e < 3.0, lo, hi)
    return torch.where(eta < 1e-8, torch.zeros_like(out), out)


def _spline(x, y):
    """Second derivatives of the not-a-knot cubic spline on a uniform grid."""
    h = x[1] - x[0]
    n = len(x)
    r = 6 * (y[2:] - 2 * y[1:-1] + y[:-2]) / h ** 2
    lo, di, up = np.ones(n - 2), np.full(n - 2, 4.0), np.ones(n - 2)
    di[0], up[0] = 6.0, 0.0
    di[-1], lo[-1] = 6.0, 0.0
    r, di = r.tolist(), di.tolist()
    for i in range(1, n - 2):
        w = lo[i] / di[i - 1]
        di[i] -= w * up[i - 1]
        r[i] -= w * r[i - 1]
    m = [0.0] * n
    m[n - 2] = r[-1] / di[-1]
    for i in range(n - 4, -1, -1):
        m[i + 1] = (r[i] - up[i] * m[i + 2]) / di[i]
    m[0], m[-1] = 2 * m[1] - m[2], 2 * m[-2] - m[-3]
    return np.array(m)


class _Uniform:
    """A cubic spline on a uniform grid from 0, its end value beyond it."""

    def __init__(self, x, y):
        m = _spline(x, y)
        self.h, self.n, self.top = float(x[1] - x[0]), len(x), float(x[-1])
        self.y, self.m = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in (y, m))
        b = np.diff(y) / self.h - self.h * (2 * m[:-1] + m[1:]) / 6
        self.slopes = np.append(b, b[-1] + self.h * (m[-2] + (m[-1] - m[-2]) / 2))

    def __call__(self, x):
        j = torch.clamp((x / self.h).long(), 0, self.n - 2)
        u = x / self.h - j
        y0, y1, m0, m1 = self.y[j], self.y[j + 1], self.m[j], self.m[j + 1]
        v = 1 - u
        out = y0 * v + y1 * u + self.h ** 2 / 6 * ((v ** 3 - v) * m0 + (u ** 3 - u) * m1)
        return torch.where(x < self.top, out, self.y[-1])


def _wgc_table(alpha, beta, gamma, m=160001):
    """K0, K1, Kq, Kx per unit prefactor on ln(eta): the bounded solution w of w'' - S w' + P w = (ab/c2) L, as two
    first-order equations, each integrated backwards exactly for a forcing linear between the points."""
    t = np.linspace(math.log(1e-5), math.log(200.0), m)
    h = t[1] - t[0]
    L = _inverse_lindhard(np.exp(t)).numpy()
    ab, sab = alpha * beta, alpha + beta
    p, c2 = 5 - 3 * sab, 1 / 36
    c1 = sab / 6 + (1 - gamma) / 36
    S, P = (c1 + c2 * (2 * p - 1)) / c2, (ab + c1 * p + c2 * p * (p - 1)) / c2
    disc = complex(S * S - 4 * P) ** 0.5
    f = ab / c2 * L

    def back(lam, g):
        e = np.exp(-lam * h)
        step = (g[:-1] * ((1 - e) / lam) + np.diff(g) / h * ((1 - e * (1 + lam * h)) / lam ** 2)).tolist()
        y, v = [0j] * m, complex(-g[-1] / lam)
        y[-1] = v
        for i in range(m - 2, -1, -1):
            v = e * v - step[i]
            y[i] = v
        return np.array(y)

    l1, l2 = (S + disc) / 2, (S - disc) / 2
    z = back(l1, f.astype(complex))
    w = back(l2, z)
    w1 = l2 * w + z
    w2 = (l2 * w1 + l1 * z + f).real
    w, w1 = w.real, w1.real
    K1 = p * w - w1
    K2 = p * (p - 1) * w - (2 * p - 1) * w1 + w2
    return t, [w, K1, (gamma - 5) / 72 * K1 + K2 / 72, (1 - gamma) / 36 * K1 + K2 / 36]


def _catmull(t, col, x):
    """Cubic (Catmull-Rom) interpolation on the uniform grid t of ln(eta); eta^2 below it."""
    c = torch.tensor(col, dtype=torch.float64, device="cuda")
    h = float(t[1] - t[0])
    lx = torch.log(torch.clamp(x, 1e-300))
    s = torch.clamp((lx - float(t[0])) / h, 0, len(t) - 2.000001)
    i = torch.clamp(s.floor().long(), 1, len(t) - 3)
    u = s - i
    y0, y1, y2, y3 = c[i - 1], c[i], c[i + 1], c[i + 2]
    v = y1 + 0.5 * u * (y2 - y0 + u * (2 * y0 - 5 * y1 + 4 * y2 - y3 + u * (3 * (y1 - y2) + y3 - y0)))
    return torch.where(lx <= float(t[0]), c[0] * (x / math.exp(t[0])) ** 2, v)


def _wgc(box, rho):
    """E and V of the second-order Wang-Govind-Carter term."""
    a, b, gamma = (5 + 5 ** 0.5) / 6, (5 - 5 ** 0.5) / 6, 2.7
    rho0 = float(rho.mean())
    C = 5 / (9 * a * b * rho0 ** (a + b - 5 / 3)) * C_TF
    eta = torch.sqrt(box.gg) / (2 * (3 * PI ** 2 * rho0) ** (1 / 3))
    t, cols = _wgc_table(a, b, gamma)
    K0, K1, Kq, Kx = (C * _catmull(t, col, eta) for col in cols)
    K1 = K1 / 6
    u = (rho - rho0) / rho0

    def fields(x):
        f0, f1, f2 = box.fwd(x), box.fwd(u * x), box.fwd(u * u * x)
        x1, x2 = box.inv(K1 * f0 + Kx * f1), box.inv(Kq * f0)
        return box.inv(K0 * f0 + K1 * f1 + Kq * f2) + u * x1 + u * u * x2, x1 + 2 * u * x2

    A, B = rho ** a, rho ** b
    sx, tx = fields(B)
    sy, ty = fields(A)
    v = a * A / rho * sx + A / rho0 * tx + b * B / rho * sy + B / rho0 * ty
    return float((A * sx).sum()) * box.dV, v


def _lmgp(box, rho):
    """E and V of the LMGP term, linear between the k_F knots (ratio 1.15), kernel of 50000 points up to 50."""
    eta = np.linspace(0.0, 50.0, 50000)
    t = torch.arange(1, 1001, dtype=torch.float64, device="cuda") / 1000
    x = torch.tensor(eta, dtype=torch.float64, device="cuda")
    x = torch.clamp(x[:, None] * t[None, :] ** (-1 / 3), eta[1] / 10, eta[-1] + 2)
    tab = ((_inverse_lindhard(x) * t ** (-1 / 6)).sum(1) * (4 / 5 * C_TF * 5 / 6 / 1000)).cpu().numpy()
    kern = _Uniform(eta, tab)
    deriv = _Uniform(eta, -eta * kern.slopes)
    a = 5 / 6
    kf = 2 * (3 * PI ** 2 * rho) ** (1 / 3)
    lo, hi = float(kf.min()), float(kf.max())
    knots = [lo * 1.15 ** i for i in range(math.ceil(math.log(hi / lo) / math.log(1.15)) + 1)]
    q = torch.sqrt(box.gg)
    ra = rho ** a
    f = box.fwd(ra)
    p1, p3, acc = torch.zeros_like(rho), torch.zeros_like(rho), torch.zeros_like(f)
    for i, k in enumerate(knots):
        # the hat function of knot i at every point
        left = (kf - knots[i - 1]) / (k - knots[i - 1]) if i else torch.ones_like(kf)
        right = (knots[i + 1] - kf) / (knots[i + 1] - k) if i + 1 < len(knots) else torch.ones_like(kf)
        w = torch.clamp(torch.minimum(left, right), 0.0, 1.0)
        K, D = kern(q / k), deriv(q / k) / k
        K.view(-1)[0] = 0.0
        D.view(-1)[0] = 0.0
        p1 += w * box.inv(K * f)
        p3 += w * box.inv(D * f)
        acc += K * box.fwd(ra * w)
    v = ra / rho * (a * p1 + a * box.inv(acc) + kf / 3 * p3)
    return float((ra * p1).sum()) * box.dV, v


def _v_loc(box, st, ph):
    """v(G) = -4 pi Z exp(-(G rc)^2 / 4) / G^2 (pi Z rc^2 at 0) times the structure factors, and per species."""
    gg = torch.where(box.gg > 0, box.gg, torch.ones_like(box.gg))
    total, each = 0, {}
    for s in sorted(set(st.symbols)):
        Z, rc = systems.SPECIES[s]
        v = torch.where(box.gg > 0, -4 * PI * Z * torch.exp(-gg * rc ** 2 / 4) / gg,
                        torch.full_like(gg, PI * Z * rc ** 2))
        each[s] = v
        w = torch.tensor([1.0 if x == s else 0.0 for x in st.symbols], dtype=torch.complex128, device="cuda")
        total = total + v * box.structure(ph, w)
    return box.inv(total * (box.N / box.vol)), each


def _ewald(st, forces=False):
    """Ion-ion energy (and forces) by direct Ewald sums converged to 64 bits."""
    q = torch.tensor(st.charges, dtype=torch.float64, device="cuda")
    R = torch.tensor(st.positions, dtype=torch.float64, device="cuda")
    eta, nat, vol = 0.35, st.nat, st.volume
    rmax, gmax = 6.2 / math.sqrt(eta), 12.4 * math.sqrt(eta)
    b = 2 * PI * np.linalg.inv(st.lattice).T
    rep = [int(math.ceil(rmax * np.linalg.norm(b[d]) / (2 * PI))) for d in range(3)]
    e = -math.sqrt(eta / PI) * float((q * q).sum()) - PI / (2 * eta * vol) * float(q.sum()) ** 2
    f = torch.zeros_like(R)
    for I in np.ndindex(*[2 * r + 1 for r in rep]):
        T = torch.tensor((np.array(I) - rep) @ st.lattice, dtype=torch.float64, device="cuda")
        d = R[:, None, :] - R[None, :, :] + T
        r = d.norm(dim=2)
        r = torch.where((r < rmax) & (r > 1e-3), r, torch.full_like(r, 1e6))
        er = torch.erfc(math.sqrt(eta) * r) / r
        qq = q[:, None] * q[None, :]
        e += 0.5 * float((qq * er).sum())
        if forces:
            g = qq * (er + 2 * math.sqrt(eta / PI) * torch.exp(-eta * r * r)) / (r * r)
            f += (g[:, :, None] * d).sum(1)
    top = [int(math.ceil(gmax * np.linalg.norm(st.lattice[d]) / (2 * PI))) for d in range(3)]
    m = [torch.arange(-t, t + 1, dtype=torch.float64, device="cuda") for t in top]
    G = torch.stack(torch.meshgrid(*m, indexing="ij"), -1).reshape(-1, 3) @ torch.tensor(b, device="cuda")
    gg = (G * G).sum(1)
    keep = (gg > 1e-12) & (gg < gmax ** 2)
    G, gg = G[keep], gg[keep]
    for c0 in range(0, len(G), 20000):
        g, w = G[c0:c0 + 20000], torch.exp(-gg[c0:c0 + 20000] / (4 * eta)) / gg[c0:c0 + 20000] * (2 * PI / vol)
        ang = R @ g.T
        cs, sn = torch.cos(ang), torch.sin(ang)
        sc, ss = q @ cs, q @ sn
        e += float((w * (sc * sc + ss * ss)).sum())
        if forces:
            f += 2 * q[:, None] * (((sn * sc - cs * ss) * w) @ g)
    return e, f


def _lda(rho):
    """Perdew-Zunger 1981: energy per particle and potential."""
    rs = (3 / (4 * PI * rho)) ** (1 / 3)
    ex = -0.75 * (3 / PI) ** (1 / 3) * rho ** (1 / 3)
    a, b, c, d, g, b1, b2 = 0.0311, -0.048, 0.0020, -0.0116, -0.1423, 1.0529, 0.3334
    lr, sq = torch.log(rs), torch.sqrt(rs)
    den = 1 + b1 * sq + b2 * rs
    ec = torch.where(rs < 1, a * lr + b + c * rs * lr + d * rs, g / den)
    vc = torch.where(rs < 1, lr * (a + 2 / 3 * c * rs) + b - a / 3 + (2 * d - c) / 3 * rs,
                     (g + 7 / 6 * g * b1 * sq + 4 / 3 * g * b2 * rs) / den ** 2)
    return ex + ec, 4 / 3 * ex + vc


def exact(case, seed):
    c = case
    if c["kind"] == "solve":
        return None                              # an iterative solution, no closed value
    st = _structure(c, seed)
    rho = _density(c, seed, st).to(torch.float64 if c["dtype"] == "fp64" else torch.float32).to(torch.float64)
    box = _Box(c, st.lattice)
    if c["kind"] == "fft":
        g = box.fwd(rho) * box.dV * torch.exp(-0.05 * box.gg).to(
            torch.float64 if c["dtype"] == "fp64" else torch.float32)
        return {"spectrum": g, "field": box.inv(g) / box.dV}
    if st.nat > 1500:
        return None                              # minutes of direct structure-factor sums
    ph = box.phases(st.scaled_positions())
    vloc, each = _v_loc(box, st, ph)
    if c["kind"] == "ions":
        e, f = _ewald(st, forces=True)
        # F_a = (1/vol) Re sum_G conj(rho(G)) v(G) (i G) exp(-i G.R_a)
        rg = box.fwd(rho).conj() * (box.dV / box.vol)
        if not box.full:
            half = torch.full((len(box.m[2]),), 2.0, dtype=torch.float64, device="cuda")
            half[0] = 1.0
            if box.n[2] % 2 == 0:
                half[-1] = 1.0
            rg = rg * half
        for s, v in each.items():
            at = [i for i, x in enumerate(st.symbols) if x == s]
            X = (rg * v).reshape(-1, len(box.m[2]))
            for i in at:
                Y = (X @ torch.stack([ph[2][i], ph[2][i] * box.m[2]], 1)).reshape(len(box.m[0]), len(box.m[1]), 2)
                Z = torch.einsum("i,ijc->jc", ph[0][i], Y)
                Z0 = torch.einsum("i,ij->j", ph[0][i] * box.m[0], Y[:, :, 0])
                dm = torch.stack([(Z0 * ph[1][i]).sum(), (Z[:, 0] * ph[1][i] * box.m[1]).sum(),
                                  (Z[:, 1] * ph[1][i]).sum()])
                f[i] += -dm.imag @ torch.tensor(box.b, device="cuda")
        return {"v_loc": vloc, "e_ion": e, "forces": f.cpu().numpy()}
    tf = C_TF * rho ** (5 / 3)
    sq = torch.sqrt(rho)
    vw = 0.5 * box.conv(sq, box.gg) / sq
    kh = torch.where(box.gg > 0, 4 * PI / torch.where(box.gg > 0, box.gg, torch.ones_like(box.gg)),
                     torch.zeros_like(box.gg))
    vh = box.conv(rho, kh)
    exc, vxc = _lda(rho)
    v = 5 / 3 * tf / rho + vw + vxc + vh + vloc
    e = float((tf + rho * (vw + exc + 0.5 * vh + vloc)).sum()) * box.dV
    if c["kedf"] == "WT":
        a, rho0 = 5 / 6, float(rho.mean())
        K = 5 / (9 * a * a) * C_TF * _inverse_lindhard(torch.sqrt(box.gg) / (2 * (3 * PI ** 2 * rho0) ** (1 / 3)))
        nl = 2 * a * rho ** (a - 1) * box.conv(rho ** a, K)
        v, e = v + nl, e + float((nl * rho).sum()) * box.dV / (2 * a)
    elif c["kedf"] in ("WGC", "LMGP"):
        en, nl = (_wgc if c["kedf"] == "WGC" else _lmgp)(box, rho)
        v, e = v + nl, e + en
    if c["dtype"] == "fp32":
        return {"potential": v}
    return {"energy": e + _ewald(st)[0], "potential": v}
