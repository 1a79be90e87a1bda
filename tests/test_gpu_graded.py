"""Vectors whose parts differ by many orders: every part keeps its own digits, whatever lies beside it.
Reference: dense numpy in FP64, on inputs scaled by powers of two where they leave its range."""
import numpy as np
import pytest

from pyprop_gb300 import _native
from test_gpu_band_shapes import _operator
from test_gpu_gram_schmidt_shapes import _handle as _diagonal
from test_gpu_solve_shapes import _dense, _handle, _rhs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tuned", [False, True])
@pytest.mark.parametrize("nl,nr,kb", [(3, 60, 6), (5, 129, 7), (6, 300, 3), (16, 500, 6)])
@pytest.mark.parametrize("fall", [0.5, 3.0])
def test_band_elementwise(tuned, nl, nr, kb, fall):
    """The operator of a handle as it comes and as the autotuner leaves it, on rows that fall by `fall` orders of ten
    per element towards one end, imaginary parts 1e-20 of the real ones: FP64 rounds each of an element's products
    and sums once, 2^-53 of its own |A| |x| each (and subnormal results to 2^-1074), numpy the two products of
    each entry."""
    import torch
    rng = np.random.default_rng(nr + kb)
    h = _native.Handle(nl, nr, _native.FP64, 4, 0, False, 0)
    h.set_overlap(1, np.tile([0.0, 1.0], nr))
    ops = _operator(h, rng, nl, nr, kb)
    h.finalize()
    if tuned:
        assert h.autotune() in (9, 10)
    g = 10.0 ** -np.minimum(fall * np.arange(nr), 300.0)
    x = rng.standard_normal((nl, nr)) + 1e-20j * rng.standard_normal((nl, nr))
    x *= np.where(np.arange(nl)[:, None] % 2, g, g[::-1])
    y = torch.zeros((nl, nr), dtype=torch.complex128, device="cuda")
    scal = [1.0, 0.37, -1.9]
    h.matvec(torch.as_tensor(x).cuda(), y, scal[1:], balanced=False)
    got, want, size, terms = y.cpu().numpy(), np.zeros((nl, nr), complex), np.zeros((2, nl, nr)), np.zeros((nl, 1))
    for td, rows, cols, M in ops:
        for r, c, A in zip(rows, cols, M):
            want[r] += scal[td] * (A @ x[c])
            a, b = abs(A.real), abs(A.imag)
            size[0, r] += abs(scal[td]) * (a @ abs(x[c].real) + b @ abs(x[c].imag))
            size[1, r] += abs(scal[td]) * (a @ abs(x[c].imag) + b @ abs(x[c].real))
            terms[r] += 2
    bound = size * 2.0 ** -53 * (3 * (2 * kb + 1) + 4 * terms + 8) + 2.0 ** -1060
    assert (abs(got.real - want.real) <= bound[0]).all() and (abs(got.imag - want.imag) <= bound[1]).all()


def test_band_nonfinite_neighbours():
    """An infinity reaches the kb elements on either side, as itself, and no other."""
    import torch
    nr = 100
    h = _native.Handle(1, nr, _native.FP64, 4, 0, False, 0)
    h.set_overlap(1, np.tile([0.0, 1.0], nr))
    h.add_potential(_native.STORAGE_DIAG, None, 2, np.ones((1, 5 * nr), dtype=np.complex128), False)
    h.finalize()
    src = torch.ones((1, nr), dtype=torch.complex128, device="cuda")
    src[0, 50] = complex(float("inf"), 1.0)
    dst = torch.zeros_like(src)
    h.matvec(src, dst, 0.0, balanced=False)
    re = dst.real[0].cpu().numpy()
    assert np.isposinf(re[48:53]).all() and (re[3:48] == 5.0).all() and (re[53:97] == 5.0).all()


@pytest.mark.parametrize("variant", [11, 12])
@pytest.mark.parametrize("nl,nr,kb", [(3, 60, 6), (5, 129, 7), (6, 300, 3)])
def test_fixed_point_window(variant, nl, nr, kb):
    """The fixed-point band forms, when asked for: an element errs by what its row's largest coefficient and the largest
    entry that its warp reads (16 or 32 elements and kb on either side) allow, 2^-58 each factor and 2^-60 for the
    part left out, and the terms' sums by 2^-53; not by what the rest of the row holds."""
    import torch
    rng = np.random.default_rng(nr + kb)
    h = _native.Handle(nl, nr, _native.FP64, 4, 0, False, 0)
    h.set_overlap(1, np.tile([0.0, 1.0], nr))
    ops = _operator(h, rng, nl, nr, kb)
    h.finalize()
    assert h.autotune(variant) == variant
    x = rng.standard_normal((nl, nr)) + 1j * rng.standard_normal((nl, nr))
    g = 10.0 ** (-0.5 * np.arange(nr))
    x *= np.where(np.arange(nl)[:, None] % 2, g, g[::-1])
    y = torch.zeros((nl, nr), dtype=torch.complex128, device="cuda")
    scal = [1.0, 0.37, -1.9]
    h.matvec(torch.as_tensor(x).cuda(), y, scal[1:], balanced=False)
    first = np.arange(nr) // (16 * (variant - 10)) * (16 * (variant - 10))
    ends = [(max(0, t - kb), t + 16 * (variant - 10) + kb) for t in first]
    big = np.maximum(abs(x.real), abs(x.imag))
    window = np.array([[row[a:b].max() for a, b in ends] for row in big])
    want, size, peak, terms = np.zeros((nl, nr), complex), np.zeros((nl, nr)), np.zeros((nl, nr)), np.zeros((nl, 1))
    for td, rows, cols, M in ops:
        for r, c, A in zip(rows, cols, M):
            want[r] += scal[td] * (A @ x[c])
            size[r] += abs(scal[td]) * ((abs(A.real) + abs(A.imag)) @ (abs(x[c].real) + abs(x[c].imag)))
            peak[r] += abs(scal[td]) * 2 * (2 * kb + 1) * np.maximum(abs(A.real), abs(A.imag)).max(axis=1) * window[c]
            terms[r] += 2
    # (two real products for each of an element's two components)
    bound = 2 * peak * (2 * 2.0 ** -58 + 2.0 ** -60) + size * 2.0 ** -53 * (2 * (2 * kb + 1) + 4 * terms + 8)
    assert (abs(y.cpu().numpy() - want) <= bound).all()


# powers of two: the rows of one problem, in turn (the last but one gives subnormal entries)
ROWS = [0, -100, 0, -130, 3, -127, -60, -61, 61, -400, 900, -1000, -20, -90, -75, -1035, 1]


@pytest.mark.parametrize("nl,nr,order", [(2, 40, 7), (9, 200, 7), (16, 129, 7), (17, 64, 4), (33, 300, 7), (64, 437, 9)])
@pytest.mark.parametrize("in_batch", [False, True])
@pytest.mark.parametrize("conj", [False, True])
def test_solve_rows_of_different_magnitude(nl, nr, order, in_batch, conj):
    """Each row by itself: its residual is summed in FP64, order + 1 terms, and the factor's inverse acts on that.
    (Subnormal entries are rounded to their spacing.)"""
    import torch
    h, U = _handle(nl, nr, order, _native.FP64)
    batch = _native.Batch([h], autotune=False) if in_batch else None     # (fewer warps per CTA)
    p = np.array([ROWS[l % len(ROWS)] for l in range(nl)])
    x = np.ldexp(1.0, p)[:, None] * _rhs(nl, nr, 3 * nl + nr)
    up = np.ldexp(1.0, -np.maximum(p, -1000))
    d = torch.as_tensor(x).cuda()
    y = torch.empty_like(d)
    h.matvec(d, y, 1.0, balanced=True)
    h.solve_sqrt_overlap(conj, d)
    cond = np.linalg.cond(U)
    tol, spacing = (order + 1) * 2.0 ** -52 * cond, 2.0 ** -1074 * up * np.sqrt(nr)
    one, both = _dense(U, x * up[:, None], conj), _dense(U, _dense(U, x * up[:, None], False), True)
    for got, want, t in ((d, one, tol), (y, both, 4 * cond * tol)):
        err = np.linalg.norm(got.cpu().numpy() * up[:, None] - want, axis=1)
        assert (err <= t * np.linalg.norm(want, axis=1) + 4 * cond ** 2 * spacing).all()
    del batch


@pytest.mark.parametrize("nl,nr,m", [(2, 30, 10), (5, 52, 20), (16, 304, 24), (9, 541, 20), (17, 1001, 24), (64, 1500, 18)])
@pytest.mark.parametrize("dorth", [False, True])
@pytest.mark.parametrize("small,rows", [(1e-12, False), (1e-30, False), (1e-60, True)])
def test_step_elementwise(nl, nr, m, dorth, small, rows):
    """A step of a diagonal operator multiplies every element by its own phase.  Every second element, or every second
    row, is small; large and small ones take turns on the spectrum, spread evenly over [-1, 1]: every beta is near 1/2
    and, with m below 2 sqrt(N / 2), the polynomials of the large points are as tame between them, so nothing
    amplifies roundings: m vectors of at most log2(N) + m roundings of 2^-53 each, for the small elements as for the
    large.  The step's polynomial is within (1/8)^m / m! of the phase."""
    import torch
    rng = np.random.default_rng(nl * nr + m)
    N = nl * nr
    weak = (np.arange(N) // (nr if rows else 1)) % 2 == 1
    line, diag = np.linspace(-1.0, 1.0, N), np.empty(N)
    order = np.argsort(np.concatenate([np.arange((~weak).sum()) * 2.0 / (~weak).sum(), np.arange(weak.sum()) * 2.0 / weak.sum() + 1e-9]))
    rank = np.empty(N, dtype=int)
    rank[order] = np.arange(N)
    diag[~weak] = rng.permutation(line[rank[:(~weak).sum()]])
    diag[weak] = rng.permutation(line[rank[(~weak).sum():]])
    x = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    x[weak] *= small
    h = _diagonal(nl, nr, m, dorth, diag)
    d = torch.as_tensor(x.reshape(nl, nr)).cuda()
    h.advance(d, np.zeros(1), 0.25)
    got, want = d.cpu().numpy().ravel(), x * np.exp(-0.25j * diag)
    for part in (weak, ~weak):
        err = np.linalg.norm(got[part] - want[part]) / np.linalg.norm(want[part])
        assert err < m * (np.log2(N) + m) * 2.0 ** -53
