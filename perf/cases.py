"""The work that a user of this framework has it do, as cases that can be timed and compared.

Every case is a hydrogen-like atom in a laser pulse (velocity gauge, m = 0): angular rows l = 0..nl-1 times nr
B-splines.  The radial matrices are formed here from the B-splines' definition, so that exact() needs none of
the framework's code; prepare() hands them to the framework as a user's program does.

Sizes and options are those of the two workload configurations (10 x 106, m = 20 and 64 x 1000, m = 30), of the
batch builder (l_max 8..64, nr 200..1500, m in 16, 24, 32), of the adjoint and bound-state tests, and odd sizes
between them.  States are smooth wave packets (a propagation starts from a bound state and stays in the part of
the spectrum that the basis resolves), fields are values of a sin^2 pulse.
"""
import math

import numpy as np
import torch

from pyprop_gb300 import LoadString, Problem, _native
from pyprop_gb300.adjoint import AdjointPropagator
from pyprop_gb300.batch import HydrogenProblem

OMEGA = 0.057


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # the small workload configuration through Problem.AdvanceSteps: one step per call, as a program that looks
        # at psi after every step does; the smallest propagation, all latency
        dict(name="problem_small", kind="problem", nl=10, nr=106, rmax=50.0, m=20, dt=0.01, steps=1, mixed=False),
        # the headline workload's size and basis (exponential-linear breakpoints), complex128 drop-in
        dict(name="advance_large", kind="advance", nl=64, nr=1000, rmax=400.0, order=7, grid="explinear", m=30,
             dt=0.001, steps=1, pulse="early", mixed=False, imag=False, dorth=False),
        # the same in the FP32-mixed form, several steps per call
        dict(name="advance_large_mixed", kind="advance", nl=64, nr=1000, rmax=400.0, order=7, grid="explinear", m=30,
             dt=0.002, steps=2, pulse="early", mixed=True, imag=False, dorth=False),
        # a mid-size problem of odd sizes, several steps per call
        dict(name="advance_ragged", kind="advance", nl=23, nr=437, rmax=170.0, order=7, grid="linear", m=24, dt=0.001,
             steps=5, pulse="early", mixed=False, imag=False, dorth=False),
        # odd sizes in the FP32-mixed form
        dict(name="advance_ragged_mixed", kind="advance", nl=37, nr=811, rmax=300.0, order=7, grid="linear", m=24,
             dt=0.002, steps=2, pulse="early", mixed=True, imag=False, dorth=False),
        # imaginary-time relaxation with renormalisation and double orthogonalisation: how a ground state is made
        dict(name="advance_relax", kind="advance", nl=16, nr=300, rmax=120.0, order=7, grid="linear", m=20, dt=0.002,
             steps=4, pulse="early", mixed=False, imag=True, dorth=True),
        # batches of uneven independent problems, one step of each
        dict(name="batch", kind="batch", count=12, nl_max=65, nr_max=1500, pick=4, mixed=False),
        dict(name="batch_mixed", kind="batch", count=24, nl_max=65, nr_max=1000, pick=11, mixed=True),
        # one application of the balanced operator at the headline size
        dict(name="matvec_large", kind="matvec", nl=64, nr=1000, rmax=400.0, order=7, grid="explinear", m=30,
             mixed=False, balanced=True),
        # Expokit: adaptive sub-steps with error control
        dict(name="expokit", kind="expokit", nl=10, nr=106, rmax=50.0, m=20, dt=0.05, steps=2),
        # a gradient of bound-state populations with respect to the pulse's samples
        dict(name="gradient", kind="gradient", nl=16, nr=200, rmax=100.0, m=20, dt=0.002, steps=6, samples=4),
        # field-free bound states of every angular row
        dict(name="bound_states", kind="bound", nl=33, nr=800, rmax=240.0, order=7),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["advance"] * 6 + ["problem", "batch", "batch", "matvec", "matvec", "expokit", "gradient", "bound"])
    if kind == "problem":
        nr = _logint(rng, 60, 160)
        return dict(kind=kind, nl=rng.randint(4, 12), nr=nr, rmax=0.47 * nr, m=rng.randint(10, 24), dt=0.01,
                    steps=rng.randint(1, 4), mixed=rng.random() < 0.4)
    if kind == "advance":
        # time steps that the Krylov space resolves: one that it does not amplifies every rounding in the stiff modes
        # at the origin, and no two programs agree on the digits; so several steps are for
        # the smaller angular ranges on even grids and for the complex64 basis
        nr = _logint(rng, 100, 1500)
        mixed, imag = rng.random() < 0.45, rng.random() < 0.2
        calm = rng.random() < 0.4
        nl = rng.randint(8, 24) if calm else _logint(rng, 8, 65)
        grid = "explinear" if nr >= 300 and not calm and rng.random() < 0.4 else "linear"
        imag = imag and calm and not mixed
        return dict(kind=kind, nl=nl, nr=nr, rmax=round(nr * rng.uniform(0.3, 0.45), 2),
                    order=7 if calm else rng.choice([7, 7, 6, 8]), grid=grid, m=rng.choice([16, 20, 24, 30, 32]),
                    dt=0.002 if mixed else 0.001, steps=rng.choice([1, 2]) if mixed else rng.randint(1, 3) if calm else 1,
                    pulse="early", mixed=mixed, imag=imag, dorth=rng.random() < 0.15)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 14), nl_max=rng.randint(12, 65), nr_max=_logint(rng, 250, 1500),
                    pick=rng.randint(0, 10 ** 6), mixed=rng.random() < 0.5)
    if kind == "matvec":
        nr = _logint(rng, 100, 1500)
        return dict(kind=kind, nl=_logint(rng, 8, 65), nr=nr, rmax=round(nr * rng.uniform(0.3, 0.45), 2),
                    order=rng.choice([7, 7, 7, 6, 8]), grid="linear", m=rng.choice([16, 30]), mixed=rng.random() < 0.4,
                    balanced=rng.random() < 0.6)
    if kind == "expokit":
        nr = _logint(rng, 60, 130)
        return dict(kind=kind, nl=rng.randint(4, 11), nr=nr, rmax=0.47 * nr, m=rng.randint(16, 24),
                    dt=round(rng.uniform(0.02, 0.06), 3), steps=rng.randint(1, 3))
    if kind == "gradient":
        nr = _logint(rng, 80, 240)
        return dict(kind=kind, nl=rng.randint(4, 20), nr=nr, rmax=0.5 * nr, m=rng.choice([16, 20]), dt=0.002,
                    steps=rng.randint(3, 6), samples=rng.randint(3, 6))
    nr = _logint(rng, 100, 900)
    return dict(kind=kind, nl=_logint(rng, 4, 33), nr=nr, rmax=round(nr * rng.uniform(0.25, 0.4), 2),
                order=rng.choice([7, 7, 6, 8]))


# ---------------------------------------------------------------------------------------------
# the operators: B-spline matrices by Gauss-Legendre quadrature, and the angular factors
# ---------------------------------------------------------------------------------------------
def _breakpoints(case):
    order, nr, rmax = case.get("order", 7), case["nr"], case["rmax"]
    n = nr - order + 4                                  # zero at both ends
    if case.get("grid", "linear") == "linear":
        return np.linspace(0.0, rmax, n)
    # exponential points on [0, 15] (gamma = 1.5), then the last gap repeated: the headline workload's grid
    n0 = max(8, (70 * n) // 997)
    e = 15.0 * (np.exp(1.5 * np.arange(n0) / (n0 - 1)) - 1.0) / (math.exp(1.5) - 1.0)
    h = (rmax - 15.0) / (n - n0)
    return np.concatenate([e, 15.0 + h * np.arange(1, n - n0 + 1)])


class _Radial:
    """Band matrices of a B-spline basis of `order` (zero at both ends): dense S, K, C2, C1, D, R and U."""

    def __init__(self, bp, order):
        kd = order - 1
        t = np.concatenate([np.full(kd, bp[0]), bp[1:-1], np.full(kd, bp[-1])])
        n = len(t) - order
        x0, w0 = np.polynomial.legendre.leggauss(order)
        a, b = bp[:-1, None], bp[1:, None]
        x = (0.5 * (b - a) * x0 + 0.5 * (a + b)).ravel()
        w = (0.5 * (b - a) * w0).ravel()
        # de Boor on a knot vector padded by one on each side (the two end splines dropped afterwards)
        tp = np.concatenate([[bp[0]], t, [bp[-1]]])
        mu = np.searchsorted(tp, x, side="right") - 1
        lev = [None, np.ones((len(x), 1))]
        for q in range(2, order + 1):
            cur = np.zeros((len(x), q))
            for j in range(q - 1):
                i = mu - q + 2 + j
                f = lev[q - 1][:, j] / (tp[i + q - 1] - tp[i])
                cur[:, j] += (tp[i + q - 1] - x) * f
                cur[:, j + 1] += (x - tp[i]) * f
            lev.append(cur)

        def diff(q, v):                                  # derivative of a combination of order-q splines' values
            out = np.zeros((len(x), q))
            for j in range(q - 1):
                i = mu - q + 2 + j
                f = (q - 1) * v[:, j] / (tp[i + q - 1] - tp[i])
                out[:, j] -= f
                out[:, j + 1] += f
            return out

        B, dB = lev[order], diff(order, lev[order - 1])
        d2B = diff(order, diff(order - 1, lev[order - 2]))
        first = mu - order                               # index (in t's numbering) of the first spline of each row
        full = np.zeros((3, len(x), n))
        for j in range(order):
            c = first + j
            ok = (c >= 0) & (c < n)
            g = np.nonzero(ok)[0]
            for k, v in enumerate((B, dB, d2B)):
                full[k, g, c[g]] = v[g, j]
        B, dB, d2B = (torch.from_numpy(f) for f in full)
        W, X = torch.from_numpy(w)[:, None], torch.from_numpy(x)[:, None]
        self.n, self.kd, self.t = n, kd, t
        self.S = B.T @ (W * B)
        self.K = -0.5 * (B.T @ (W * d2B))
        self.K = 0.5 * (self.K + self.K.T)
        self.C2 = B.T @ (W / (2.0 * X * X) * B)
        self.C1 = -(B.T @ (W / X * B))
        self.D = B.T @ (W * dB)
        self.D = 0.5 * (self.D - self.D.T)
        self.R = -self.C1
        self.U = torch.linalg.cholesky(self.S).T.contiguous()

    def band(self, M, upper=False):
        """BLAS band storage, element (i, j) at j * width + kb + i - j (upper: the upper triangle only)."""
        kd, n, M = self.kd, self.n, M.numpy()
        width = kd + 1 if upper else 2 * kd + 1
        out = np.zeros(n * width)
        for d in range(0 if upper else -kd, kd + 1):     # j = i + d
            i = np.arange(max(0, -d), min(n, n - d))
            out[(i + d) * width + kd - d] = M[i, i + d]
        return out

    def diagonals(self, M):
        kd, n, M = self.kd, self.n, M.numpy()
        out = np.zeros((2 * kd + 1, n))
        for d in range(-kd, kd + 1):
            i = np.arange(max(0, -d), min(n, n - d))
            out[d + kd, i] = M[i, i + d]
        return out

    def greville(self):
        return np.array([self.t[i + 1:i + self.kd + 1].mean() for i in range(self.n)])


_RADIAL = {}


def _radial(case):
    key = (case.get("order", 7), case["nr"], case["rmax"], case.get("grid", "linear"))
    if key not in _RADIAL:
        if len(_RADIAL) > 40:
            _RADIAL.clear()
        _RADIAL[key] = _Radial(_breakpoints(case), key[0])
    return _RADIAL[key]


def _dipole(nl):
    """(row, col) pairs of the dipole selection rule and the factors of D and R in <row| d/dz |col>."""
    pairs, cD, cR = [], [], []
    for l in range(nl):
        for k in (l - 1, l + 1):
            if 0 <= k < nl:
                lo = min(l, k)
                c = (lo + 1.0) / math.sqrt((2 * lo + 1.0) * (2 * lo + 3.0))
                pairs.append((l, k))
                cD.append(c)
                cR.append(-(k + 1) * c if l > k else k * c)
    return np.array(pairs, dtype=np.int32), np.array(cD), np.array(cR)


def _handle(case, m, mixed, dorth=False):
    """A finalized handle for the case's operator, as PamPropagator.SetupStep makes it."""
    rad, nl = _radial(case), case["nl"]
    K, C2, C1, D, R = (rad.band(M) for M in (rad.K, rad.C2, rad.C1, rad.D, rad.R))
    ll = np.arange(nl) * (np.arange(nl) + 1.0)
    pairs, cD, cR = _dipole(nl)
    prec = _native.FP32_MIXED if mixed else _native.FP64
    h = _native.Handle(nl, case["nr"], prec, m, 0, dorth, torch.cuda.current_stream().cuda_stream)
    h.set_overlap(rad.kd, rad.band(rad.U, upper=True))
    h.add_potential(_native.STORAGE_DIAG, None, rad.kd, (K + C1)[None] + ll[:, None] * C2[None], False)
    h.add_potential(_native.STORAGE_SIMP, pairs, rad.kd, -1j * (cD[:, None] * D[None] + cR[:, None] * R[None]), True)
    h.finalize()
    return h


# ---------------------------------------------------------------------------------------------
# states and fields
# ---------------------------------------------------------------------------------------------
_FILTER = {}


def _filter(case):
    """Banded Cholesky factors of H_l + 2 S for every row l: rows L(i, i - kd .. i) and columns L(i + 1 .. i + kd, i)."""
    rad, nl = _radial(case), case["nl"]
    if (id(rad), nl) not in _FILTER:
        kd, n = rad.kd, rad.n
        ll = np.arange(nl) * (np.arange(nl) + 1.0)
        A0, C2 = rad.diagonals(rad.K + rad.C1 + 2.0 * rad.S), rad.diagonals(rad.C2)
        A = A0[:, :, None] + ll * C2[:, :, None]          # A[m, i] = H(i, i - kd + m) per row l, m <= kd
        rows = np.zeros((n + kd, kd + 1, nl))
        rows[:kd, kd] = 1.0                               # rows before the first: no coupling
        for i in range(n):
            w, li = rows[i:i + kd], rows[i + kd]
            for m in range(kd):
                v = A[m, i].copy()
                for p in range(m):
                    v -= li[p] * w[m, p + kd - m]
                li[m] = v / w[m, kd] if i - kd + m >= 0 else 0.0
            li[kd] = np.sqrt(A[kd, i] - np.sum(li[:kd] ** 2, axis=0))
        rows = rows[kd:]
        cols = np.zeros((n, kd, nl))
        for m in range(kd):
            cols[:n - 1 - m, m] = rows[1 + m:, kd - 1 - m]
        if len(_FILTER) > 40:
            _FILTER.clear()
        _FILTER[(id(rad), nl)] = (rad, rows, cols)
    return _FILTER[(id(rad), nl)][1:]


def _state(case, seed):
    """Smooth wave packets, S-normalised: spline coefficients are a function's values at the Greville points, with
    weights falling with l as a pulse's first cycles leave them, then (H_l + 2)^-1 four times: what a propagation from
    a bound state holds is the low end of the spectrum, not the stiff modes at the origin."""
    rad, nl, rmax = _radial(case), case["nl"], case["rmax"]
    kd, n = rad.kd, rad.n
    rng = np.random.default_rng([seed, nl, case["nr"]])
    r = rad.greville()
    l = np.arange(nl)[:, None]
    out = np.zeros((nl, n), dtype=complex)
    for _ in range(4):
        c, s, k = rng.uniform(1.0, 0.45 * rmax), rng.uniform(3.0, 8.0), rng.uniform(-0.7, 0.7)
        a = (rng.standard_normal(nl) + 1j * rng.standard_normal(nl))[:, None]
        out += a * np.exp(-0.5 * ((r - c) / s) ** 2 + 1j * k * r)
    out += 3.0 * rng.standard_normal((nl, 1)) * np.exp(-r / 2.0)     # the part that stayed bound
    out *= (r / (r + 2.0)) ** (l + 1.0) * np.exp(-(r / (0.8 * rmax)) ** 8) * np.exp(-l / 6.0)
    rows, cols = _filter(case)
    S = rad.S.numpy()
    for _ in range(4):
        z = np.zeros((n + 2 * kd, nl), dtype=complex)
        b = (out @ S).T
        for i in range(n):
            z[i + kd] = (b[i] - np.sum(rows[i, :kd] * z[i:i + kd], axis=0)) / rows[i, kd]
        for i in reversed(range(n)):
            z[i + kd] = (z[i + kd] - np.sum(cols[i] * z[i + kd + 1:i + 2 * kd + 1], axis=0)) / rows[i, kd]
        out = z[kd:n + kd].T.copy()
    return out / math.sqrt(np.real(np.sum(out.conj() * (out @ S))))


def _fields(seed, n, dt, pulse="peak"):
    """n consecutive values of A(t) from a seeded time on: in the pulse's first cycles, or anywhere under its envelope."""
    rng = np.random.default_rng([seed, 77])
    T = 2 * math.pi / OMEGA * 8
    t = (rng.uniform(0.005, 0.03) if pulse == "early" else rng.uniform(0.1, 0.9)) * T + np.arange(n) * dt
    return 0.1 / OMEGA * np.sin(math.pi * t / T) ** 2 * -np.cos(OMEGA * t)


def _case_fields(case, seed):
    return _fields(seed, case.get("steps", 1), case.get("dt", 0.005), case.get("pulse", "peak"))


def _dt(case):
    return complex(0.0, -case["dt"]) if case.get("imag") else complex(case["dt"])


def _batch_members(case):
    rng = np.random.default_rng([case["pick"], case["count"]])
    out = []
    for _ in range(case["count"]):
        nr = int(rng.integers(200, case["nr_max"] + 1))
        out.append(dict(nl=int(rng.integers(9, case["nl_max"] + 1)), nr=nr, rmax=round(float(rng.uniform(0.3, 0.45)) * nr, 2),
                        order=7, grid="linear", m=int(rng.choice([16, 24, 32])), mixed=case["mixed"],
                        dt=0.002 if case["mixed"] else 0.001, steps=1, pulse="early"))
    return out


_INI = """
[Representation]
rank = 2
type = core.CombinedRepresentation_2
representation0 = "AngularRepresentation"
representation1 = "RadialRepresentation"

[AngularRepresentation]
type = core.ReducedSphericalHarmonicRepresentation
maxl = %(lmax)d
m = 0

[RadialRepresentation]
type = core.BSplineRepresentation
xmin = 0.0
xmax = %(rmax)r
xsize = %(nbreak)d
bpstype = 'linear'
continuity = 'zero'
order = 7
quad_order_additional = 0
projection_algorithm = 0

[PulseParameters]
frequency = 0.057
cycles = 8
pulse_duration = 2 * pi / frequency * cycles
amplitude = 0.05 / frequency

[Propagation]
base = "PulseParameters"
potential_evaluation = []
grid_potential_list = ["RadialKineticEnergy", "AngularKineticEnergy", "CoulombPotential", "LaserPotentialVelocity1", "LaserPotentialVelocity2", "LaserPotentialVelocity3"]
propagator = PamPropagator
base_propagator = BasisPropagator
timestep = %(dt)r
duration = 5.0
renormalization = False
krylov_basis_size = %(m)d
krylov_exponentiation_method = 0
krylov_double_orthogonalization = False
krylov_precision = "%(precision)s"
silent = True

[RadialKineticEnergy]
classname = "KineticEnergyPotential"
geometry0 = "Diagonal"
geometry1 = "banded-nonhermitian"
differentiation0 = 0
differentiation1 = 2
mass = 1

[AngularKineticEnergy]
classname = "AngularKineticEnergyPotential"
geometry0 = "Diagonal"
geometry1 = "banded-nonhermitian"
mass = 1
angular_rank = 0
radial_rank = 1

[CoulombPotential]
classname = "RadialCoulombPotential"
geometry0 = "Diagonal"
geometry1 = "banded-nonhermitian"
angular_rank = 0
radial_rank = 1

[LaserPotentialVelocityBase]
base = "PulseParameters"
geometry0 = "dipoleselectionrule"
geometry1 = "banded-nonhermitian"
angular_rank = 0
radial_rank = 1
time_function = LaserFunctionVelocity
charge = -1.0

[LaserPotentialVelocity1]
base = "LaserPotentialVelocityBase"
classname = "DipoleLaserPotentialVelocityRadialDerivative"
differentiation1 = 1

[LaserPotentialVelocity2]
base = "LaserPotentialVelocityBase"
classname = "DipoleLaserPotentialVelocityAngularDerivative"
differentiation0 = 1

[LaserPotentialVelocity3]
base = "LaserPotentialVelocityBase"
classname = "DipoleLaserPotentialVelocity"
"""


def _problem_start(seed):
    """The time at which a problem case's steps begin, inside the pulse."""
    return float(np.random.default_rng([seed, 3]).uniform(0.1, 0.9)) * 2 * math.pi / OMEGA * 8


def _problem_fields(seed, n, dt):
    T = 2 * math.pi / OMEGA * 8
    t, out = _problem_start(seed), []
    for _ in range(n):
        out.append(0.05 / OMEGA * math.sin(math.pi * t / T) ** 2 * -math.cos(OMEGA * t))
        t = t + dt
    return np.array(out)


def _bound_bands(case, seed):
    """Symmetric bands (row, diagonal, i) of H_l of a one-electron model -(1 + (Z - 1) e^(-a r)) / r, as Z C1 - ...:
    a seeded mixture of the kinetic, centrifugal and Coulomb matrices."""
    rad = _radial(case)
    z = float(np.random.default_rng([seed, 5]).uniform(0.8, 1.6))
    K, C2, C1, S = (rad.diagonals(M) for M in (rad.K, rad.C2, rad.C1, rad.S))
    ll = np.arange(case["nl"]) * (np.arange(case["nl"]) + 1.0)
    return (K + z * C1)[None] + ll[:, None, None] * C2[None], S


def _max_states(case):
    return 24


def _gradient_inputs(case, seed):
    rad, nl = _radial(case), case["nl"]
    rng = np.random.default_rng([seed, 11])
    samples = rng.uniform(-0.9, 0.9, case["samples"])
    Li = torch.linalg.inv(rad.U)
    states = []
    for l in range(min(2, nl)):
        H = rad.K + rad.C1 + l * (l + 1.0) * rad.C2
        _, v = torch.linalg.eigh(Li.T @ (0.5 * (H + H.T)) @ Li)
        c = (Li @ v[:, :2]).T.numpy()
        for row in c:
            phi = np.zeros((nl, case["nr"]), dtype=complex)
            phi[l] = row
            states.append(phi.ravel())
    return samples, np.array(states)


# ---------------------------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "problem":
        conf = LoadString(_INI % dict(lmax=case["nl"] - 1, rmax=case["rmax"], nbreak=case["nr"] - 3, m=case["m"], dt=case["dt"],
                                      precision="fp32-mixed" if case["mixed"] else "fp64"))
        prob = Problem(conf, device="cuda")
        prob.SetupStep()
        psi = torch.as_tensor(_state(case, seed)).to("cuda", prob.psi.data.dtype)
        return dict(case=case, prob=prob, psi=psi, t0=_problem_start(seed))
    if kind == "advance":
        h = _handle(case, case["m"], case["mixed"], case["dorth"])
        h.set_renormalization(case["imag"])
        h.autotune()
        psi = torch.as_tensor(_state(case, seed)).to("cuda", torch.complex64 if case["mixed"] else torch.complex128)
        return dict(case=case, h=h, psi=psi, out=torch.empty_like(psi), f=_case_fields(case, seed))
    if kind == "batch":
        ms = _batch_members(case)
        hs = [_handle(c, c["m"], case["mixed"]) for c in ms]
        dtype = torch.complex64 if case["mixed"] else torch.complex128
        psi = [torch.as_tensor(_state(c, seed + k)).to("cuda", dtype) for k, c in enumerate(ms)]
        b = _native.Batch(hs, autotune=True, stream=torch.cuda.current_stream().cuda_stream)
        return dict(case=case, batch=b, psi=psi, out=[torch.empty_like(p) for p in psi],
                    f=np.array([_case_fields(c, seed + k) for k, c in enumerate(ms)]), dts=[c["dt"] for c in ms])
    if kind == "matvec":
        h = _handle(case, case["m"], case["mixed"])
        h.autotune()
        psi = torch.as_tensor(_state(case, seed)).to("cuda", torch.complex64 if case["mixed"] else torch.complex128)
        return dict(case=case, h=h, psi=psi, out=torch.empty_like(psi), f=_case_fields(case, seed))
    if kind == "expokit":
        h = _handle(case, case["m"] + 1, False, True)
        h.autotune()
        psi = torch.as_tensor(_state(case, seed)).cuda()
        return dict(case=case, h=h, psi=psi, out=torch.empty_like(psi), f=_case_fields(case, seed))
    if kind == "gradient":
        hp = HydrogenProblem(lmax=case["nl"] - 1, nr=case["nr"], rmax=case["rmax"], m=case["m"], dt=case["dt"], setup="gpu")
        samples, states = _gradient_inputs(case, seed)
        return dict(case=case, prop=AdjointPropagator(hp, case["steps"], case["samples"]), psi=_state(case, seed),
                    samples=samples, states=states)
    H, S = _bound_bands(case, seed)
    return dict(case=case, H=torch.as_tensor(H).cuda(), S=torch.as_tensor(S).cuda())


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "problem":
        prob = s["prob"]
        prob.psi.data.copy_(s["psi"])
        prob.PropagatedTime = s["t0"]
        prob.AdvanceSteps(case["steps"])
        return {"psi": prob.psi.data}
    if kind == "advance":
        s["out"].copy_(s["psi"])
        s["h"].advance(s["out"], s["f"], _dt(case))
        return {"psi": s["out"]}
    if kind == "batch":
        torch._foreach_copy_(s["out"], s["psi"])
        s["batch"].advance(s["out"], s["f"], s["dts"])
        return {"psi": s["out"]}
    if kind == "matvec":
        if case["balanced"]:
            s["h"].matvec(s["psi"], s["out"], s["f"], balanced=True)
        else:                                            # S^-1 H psi, BasisPropagator.MultiplyHamiltonian
            s["h"].matvec(s["psi"], s["out"], s["f"], balanced=False)
            s["h"].solve_sqrt_overlap(True, s["out"])
            s["h"].solve_sqrt_overlap(False, s["out"])
        return {"out": s["out"]}
    if kind == "expokit":
        s["out"].copy_(s["psi"])
        s["h"].expokit_advance(s["out"], s["f"], case["dt"], 1e-10, 100.0)
        return {"psi": s["out"]}
    if kind == "gradient":
        psi = s["prop"].forward(s["psi"], s["samples"])
        grad, per_step = s["prop"].gradient(psi, s["states"])
        return {"psi": psi, "grad": grad, "per_step": per_step}
    counts, energies, vectors = _native.bound_states(s["H"], s["S"], 0.0, _max_states(case))
    return {"counts": counts, "energies": energies, "vectors": vectors}


# ---------------------------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------------------------
def _matvec_flops(c):
    # one band of 2 kd + 1 real coefficients per stored slot on complex vectors, and two kd-band solves
    kd = c.get("order", 7) - 1
    slots = c["nl"] + 2 * (c["nl"] - 1)
    return 4.0 * (2 * kd + 1) * slots * c["nr"] + 2 * 4.0 * (kd + 1) * c["nl"] * c["nr"]


def _operator_bytes(c):
    kd = c.get("order", 7) - 1
    return 8.0 * ((2 * kd + 1) * (3 * c["nl"] - 2) + kd + 1) * c["nr"]


def _step_flops(c, m):
    N = c["nl"] * c["nr"]
    return m * _matvec_flops(c) + 16.0 * N * m * (m + 1) / 2 + 8.0 * N * m


def work(case):
    kind = case["kind"]
    if kind == "batch":
        es, parts = (8 if case["mixed"] else 16), _batch_members(case)
        return {"bytes": sum(_operator_bytes(c) + 2.0 * es * c["nl"] * c["nr"] for c in parts),
                "flops": sum(_step_flops(c, c["m"]) for c in parts)}
    N = case["nl"] * case["nr"]
    if kind == "bound":
        kd = case["order"] - 1
        # the bands read once, the vectors written; one factorisation and three solves per state (about three a row)
        return {"bytes": 8.0 * (2 * kd + 1) * (case["nl"] + 1) * case["nr"] + 8.0 * case["nl"] * _max_states(case) * case["nr"],
                "flops": 3.0 * N * (2.0 * kd * kd + 3 * 8.0 * kd)}
    es = 8.0 if case.get("mixed") else 16.0
    b = _operator_bytes(case) + 2 * es * N
    if kind == "matvec":
        return {"bytes": b, "flops": _matvec_flops(case)}
    if kind == "expokit":
        return {"bytes": b, "flops": case["steps"] * _step_flops(case, case["m"] + 1)}
    if kind == "gradient":
        # per step: forward twice (once recomputed), the co-state, and the operator of twice the rows and vectors
        return {"bytes": b, "flops": case["steps"] * (3 * _step_flops(case, case["m"]) + 2 * _step_flops(case, min(2 * case["m"], 45)))}
    return {"bytes": b, "flops": case["steps"] * _step_flops(case, case["m"])}


# ---------------------------------------------------------------------------------------------
# the same in 64 bits, by plain torch on the host
# ---------------------------------------------------------------------------------------------
class _Plain:
    """H(f) and the overlap factor of a case as dense radial matrices acting on (rows, nr) complex128."""

    def __init__(self, case):
        self.rad, nl = _radial(case), case["nl"]
        self.nl = nl
        self.M = torch.cat([self.rad.K + self.rad.C1, self.rad.C2, self.rad.D, self.rad.R]).to(torch.float64)
        self.ll = torch.arange(nl, dtype=torch.float64) * (torch.arange(nl) + 1.0)
        pairs, cD, cR = _dipole(nl)
        self.AD, self.AR = torch.zeros(nl, nl, dtype=torch.float64), torch.zeros(nl, nl, dtype=torch.float64)
        for (i, j), d, r in zip(pairs, cD, cR):
            self.AD[i, j], self.AR[i, j] = d, r

    @staticmethod
    def _cols(x):                                        # (rows, nr) complex -> (nr, 2 rows) real
        return torch.cat([x.real, x.imag]).T.contiguous()

    @staticmethod
    def _back(y):
        y = y.T
        n = y.shape[0] // 2
        return torch.complex(y[:n].contiguous(), y[n:].contiguous())

    def H(self, x, f, parts=(True, True)):
        y = self.M @ self._cols(x)
        n = self.rad.n
        out = torch.zeros_like(x)
        if parts[0]:
            out += self._back(y[:n]) + self.ll[:, None] * self._back(y[n:2 * n])
        if parts[1]:
            out += -1j * f * (self.AD.to(x.dtype) @ self._back(y[2 * n:3 * n]) + self.AR.to(x.dtype) @ self._back(y[3 * n:]))
        return out

    def mulU(self, x):
        return self._back(self.rad.U @ self._cols(x))

    def solve(self, x, conj):
        A = self.rad.U.T if conj else self.rad.U
        return self._back(torch.linalg.solve_triangular(A, self._cols(x), upper=not conj))

    def balanced(self, x, f):
        return self.solve(self.H(self.solve(x, False), f), True)

    def S(self, x):
        return self._back(self.rad.S @ self._cols(x))


class _Doubled(_Plain):
    """[[A, A1], [0, A]] acting on [u; v]: the step's derivative with respect to the field value."""

    def H(self, x, f, parts=(True, True)):
        u, v = x[:self.nl], x[self.nl:]
        return torch.cat([_Plain.H(self, u, f) + _Plain.H(self, v, 1.0, (False, True)), _Plain.H(self, v, f)])


def _pade(H, dt):
    """First column of exp(-i dt H): diagonal Pade (6, 6) with scaling and squaring."""
    A = -1j * dt * H
    mx = float(A.abs().max())
    s = max(0, math.ceil(math.log2(mx))) if mx > 0 else 0
    A = A / 2.0 ** s
    c = [1.0]
    for i in range(6):
        c.append(c[-1] * (6 - i) / ((i + 1) * (12 - i)))
    I = torch.eye(len(A), dtype=A.dtype)
    A2 = A @ A
    P = A @ (c[1] * I + A2 @ (c[3] * I + c[5] * A2))
    Q = c[0] * I + A2 @ (c[2] * I + A2 @ (c[4] * I + c[6] * A2))
    E = I + 2.0 * torch.linalg.solve(Q - P, P)
    for _ in range(s):
        E = E @ E
    return E[:, 0]


def _step(op, x, f, m, dt, renorm=False, dorth=False):
    """One Krylov step in balanced coordinates: classical Gram-Schmidt Arnoldi, Pade exponential."""
    shape = x.shape
    beta0 = torch.linalg.vector_norm(x)
    V = torch.zeros((m, x.numel()), dtype=x.dtype)
    H = torch.zeros((m, m), dtype=x.dtype)
    V[0] = (x / beta0).reshape(-1)
    for J in range(m):
        w = op.balanced(V[J].reshape(shape), f).reshape(-1)
        h = V[:J + 1].conj() @ w
        w = w - h @ V[:J + 1]
        if dorth:
            h2 = V[:J + 1].conj() @ w
            w = w - h2 @ V[:J + 1]
            h = h + h2
        H[:J + 1, J] = h
        if J + 1 < m:
            b = torch.linalg.vector_norm(w)
            if b < math.sqrt(np.finfo(float).eps):
                H, V = H[:J + 1, :J + 1], V[:J + 1]
                break
            H[J + 1, J] = b
            V[J + 1] = w / b
    y = _pade(H, dt)
    x = (beta0 * (y @ V)).reshape(shape)
    return x / torch.linalg.vector_norm(x) if renorm else x


def _propagate(case, m, psi, fields, dt, renorm=False, dorth=False, cls=_Plain):
    op = cls(case)
    x = op.mulU(psi)
    for f in fields:
        x = _step(op, x, float(f), m, dt, renorm, dorth)
    return op.solve(x, False)


def _start(case, seed):
    psi = torch.as_tensor(_state(case, seed))
    return psi.to(torch.complex64).to(torch.complex128) if case.get("mixed") else psi


def exact(case, seed):
    kind = case["kind"]
    if kind == "problem":
        return {"psi": _propagate(case, case["m"], _start(case, seed), _problem_fields(seed, case["steps"], case["dt"]), case["dt"])}
    if kind == "advance":
        return {"psi": _propagate(case, case["m"], _start(case, seed), _case_fields(case, seed), _dt(case),
                                  case["imag"], case["dorth"])}
    if kind == "batch":
        out = []
        for k, c in enumerate(_batch_members(case)):
            out.append(_propagate(c, c["m"], _start(c, seed + k), _case_fields(c, seed + k), c["dt"]))
        return {"psi": out}
    if kind == "matvec":
        op, psi, f = _Plain(case), _start(case, seed), float(_case_fields(case, seed)[0])
        if case["balanced"]:
            return {"out": op.balanced(psi, f)}
        return {"out": op.solve(op.solve(op.H(psi, f), True), False)}
    if kind == "expokit":
        # the exponential itself, from the eigenvectors of the dense balanced operator
        op = _Plain(case)
        x = op.mulU(_start(case, seed))
        n = x.numel()
        Ui = torch.linalg.inv(op.rad.U)
        blocks = [Ui.T @ M @ Ui for M in (op.rad.K + op.rad.C1, op.rad.C2, op.rad.D, op.rad.R)]
        H0 = torch.kron(torch.eye(op.nl, dtype=torch.float64), blocks[0]) + torch.kron(torch.diag(op.ll), blocks[1])
        H1 = torch.kron(op.AD, blocks[2]) + torch.kron(op.AR, blocks[3])
        for f in _case_fields(case, seed):
            H = torch.complex(H0, -float(f) * H1)
            e, v = torch.linalg.eigh(0.5 * (H + H.conj().T))
            x = (v @ (torch.exp(-1j * case["dt"] * e) * (v.conj().T @ x.reshape(n)))).reshape(x.shape)
        return {"psi": op.solve(x, False)}
    if kind == "gradient":
        return _exact_gradient(case, seed)
    H, S = _bound_bands(case, seed)
    rad = _radial(case)
    z = float(np.random.default_rng([seed, 5]).uniform(0.8, 1.6))
    Ui = torch.linalg.inv(rad.U)
    counts = np.zeros(case["nl"], dtype=np.int32)
    energies = np.zeros((case["nl"], _max_states(case)))
    for l in range(case["nl"]):
        A = Ui.T @ (rad.K + z * rad.C1 + l * (l + 1.0) * rad.C2) @ Ui
        e = torch.linalg.eigvalsh(0.5 * (A + A.T)).numpy()
        counts[l] = int((e < 0.0).sum())
        k = min(int(counts[l]), _max_states(case))
        energies[l, :k] = e[:k]
    return {"counts": counts, "energies": energies, "vectors": None}


def _exact_gradient(case, seed):
    """The discrete adjoint of bound-state populations with respect to a piecewise-linear field's samples."""
    samples, states = _gradient_inputs(case, seed)
    n, k, dt, m = case["steps"], case["samples"], case["dt"], case["m"]
    W = np.zeros((n, k))
    for i in range(n):
        x = i * dt / (n * dt) * (k - 1)
        j = min(int(math.floor(x)), k - 2)
        W[i, j] += 1.0 - (x - j)
        W[i, j + 1] += x - j
    f = W @ samples
    op, two = _Plain(case), _Doubled(case)
    phi = torch.as_tensor(states)
    psi = [torch.as_tensor(_state(case, seed))]
    for i in range(n):
        psi.append(op.solve(_step(op, op.mulU(psi[-1]), float(f[i]), m, dt), False))
    amps = phi.conj() @ op.S(psi[-1]).reshape(-1)
    gamma = (phi.T @ amps).reshape(psi[0].shape)
    d = np.zeros(n)
    for i in reversed(range(n)):
        aug = torch.cat([torch.zeros_like(psi[i]), psi[i]])
        x = torch.cat([op.mulU(aug[:op.nl]), op.mulU(aug[op.nl:])])
        x = _step(two, x, float(f[i]), min(2 * m, 45), dt)
        dpsi = op.solve(x[:op.nl], False)
        d[i] = 2.0 * float(torch.sum(gamma.conj() * op.S(dpsi)).real)
        gamma = op.solve(_step(op, op.mulU(gamma), float(f[i]), m, -dt), False)
    return {"psi": psi[-1], "grad": W.T @ d, "per_step": d}
