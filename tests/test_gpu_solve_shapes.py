"""The overlap-factor solves at the edges of their shapes: radial sizes around the tiles, blocks and
halos, row counts around the row groups, every band width, pinned chunk counts, and right-hand sides
outside FP32's exponent range or falling by many orders towards the origin.  Reference: dense
substitution in FP64 (numpy)."""
import numpy as np
import pytest

from pyprop_gb300 import _native
from pyprop_gb300.basis import bspline as bs

pytestmark = pytest.mark.gpu


def _factor(nr, order):
    nb = nr - order + 4
    basis = bs.BSplineBasis(bs.linear_breakpoints(0.0, 0.4 * nr, nb), order, bs.continuity_sequence(nb, order, "zero"))
    assert basis.count == nr
    kd = order - 1
    Ud = bs.band_cholesky_upper_diagonals(basis.band_diagonals(np.ones(len(basis.grid)), 0), kd)
    U = np.zeros((nr, nr))
    band = np.zeros(nr * (kd + 1))
    for d in range(kd + 1):
        i = np.arange(nr - d)
        U[i, i + d] = Ud[d, : nr - d]
        band[(i + d) * (kd + 1) + kd - d] = Ud[d, : nr - d]
    return U, band, kd


def _handle(nl, nr, order, precision):
    """A handle whose operator is the identity, so that its balanced form is U^-T U^-1."""
    U, band, kd = _factor(nr, order)
    one = np.zeros((1, (2 * kd + 1) * nr), dtype=np.complex128)
    one[0, np.arange(nr) * (2 * kd + 1) + kd] = 1.0
    h = _native.Handle(nl, nr, precision, 2, 0, False, 0)
    h.set_overlap(kd, band)
    h.add_potential(_native.STORAGE_IDENT, None, kd, one, False)
    h.finalize()
    return h, U


def _dense(U, x, conj):
    import scipy.linalg as sl
    return sl.solve_triangular(U, x.T, trans="T" if conj else "N").T


def _rhs(nl, nr, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((nl, nr)) + 1j * rng.standard_normal((nl, nr))


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


SHAPES = [(1, 9, 7), (3, 16, 7), (4, 17, 7), (5, 33, 7), (9, 64, 7), (2, 127, 7), (16, 128, 7), (17, 129, 7), (33, 300, 7),
          (64, 437, 7), (65, 1500, 7), (3, 40, 2), (4, 61, 3), (7, 90, 4), (8, 111, 5), (13, 112, 6), (21, 113, 8),
          (31, 251, 9)]


@pytest.mark.parametrize("nl,nr,order", SHAPES)
@pytest.mark.parametrize("conj", [False, True])
def test_fp64_solve(nl, nr, order, conj):
    import torch
    h, U = _handle(nl, nr, order, _native.FP64)
    x = _rhs(nl, nr, 1000 * nl + nr)
    want = _dense(U, x, conj)
    d = torch.as_tensor(x).cuda()
    h.solve_sqrt_overlap(conj, d)
    assert _rel(d.cpu().numpy(), want) < 1e-14 * max(1.0, np.linalg.cond(U) / 10)


@pytest.mark.parametrize("chunks", [1, 2, 3, 7, 19])
@pytest.mark.parametrize("precision", [_native.FP64, _native.FP32_MIXED])
def test_pinned_chunks(monkeypatch, chunks, precision):
    """Every chunking gives the same balanced operator U^-T U^-1 (complex64: its two intermediate
    vectors and the result rounded once each, 2^-24 of an entry, times what the second solve amplifies)."""
    import torch
    monkeypatch.setenv("GBPROP_SOLVE_CHUNKS", "%d,%d" % (chunks, chunks))
    h, U = _handle(11, 299, 7, precision)
    h.autotune()
    x = _rhs(11, 299, 5)
    cdt = torch.complex128 if precision == _native.FP64 else torch.complex64
    d = torch.as_tensor(x).to("cuda", cdt)
    y = torch.empty_like(d)
    h.matvec(d, y, 1.0, balanced=True)
    want = _dense(U, _dense(U, d.cpu().numpy().astype(np.complex128), False), True)
    tol = 1e-13 if precision == _native.FP64 else 2.0 ** -24 * (1 + 2 * np.linalg.cond(U))
    assert _rel(y.cpu().numpy().astype(np.complex128), want) < tol


@pytest.mark.parametrize("chunks", [(1, 2), (3, 7), (19, 1)])
@pytest.mark.parametrize("precision", [_native.FP64, _native.FP32_MIXED])
def test_pinned_chunks_are_used(monkeypatch, chunks, precision):
    """(299 elements split into chunks of 304, 160, 112, 48 and 16: multiples of sixteen)"""
    monkeypatch.setenv("GBPROP_SOLVE_CHUNKS", "%d,%d" % chunks)
    h, _ = _handle(11, 299, 7, precision)
    h.autotune()
    assert tuple(h.tuning()[1]) == chunks


@pytest.mark.parametrize("scale", [1e-300, 1e-60, 1e-25, 1e25, 1e60, 1e300])
def test_fp64_solve_exponent_range(scale):
    import torch
    h, U = _handle(5, 200, 7, _native.FP64)
    x = _rhs(5, 200, 9)
    want = _dense(U, x, False)
    d = torch.as_tensor(x * scale).cuda()
    h.solve_sqrt_overlap(False, d)
    assert _rel(d.cpu().numpy() / scale, want) < 1e-13


@pytest.mark.parametrize("conj", [False, True])
def test_fp64_solve_graded(conj):
    """A right-hand side that falls by twelve orders towards one end: every hundred elements keep
    their own digits (the inverse band drops 2^-26 of a row; against values 11 times larger per band width three passes leave
    (11 2^-26)^3)."""
    import torch
    h, U = _handle(3, 600, 7, _native.FP64)
    fall = 10.0 ** (-12.0 * np.arange(600) / 599)
    x = _rhs(3, 600, 11) * (fall if conj else fall[::-1])
    want = _dense(U, x, conj)
    d = torch.as_tensor(x).cuda()
    h.solve_sqrt_overlap(conj, d)
    got = d.cpu().numpy()
    for i in range(0, 600, 100):
        assert _rel(got[:, i:i + 100], want[:, i:i + 100]) < 1e-12


def test_zero_and_nonfinite():
    import torch
    h, _ = _handle(3, 200, 7, _native.FP64)
    d = torch.zeros((3, 200), dtype=torch.complex128, device="cuda")
    h.solve_sqrt_overlap(False, d)
    assert not bool(d.abs().max())
    d[1, 150] = complex(float("nan"), 0.0)
    h.solve_sqrt_overlap(False, d)
    assert bool(torch.isnan(d.real[1, 150])) and bool((d[0] == 0).all())
