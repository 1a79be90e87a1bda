"""The term-per-warp band kernels (variants 9 and 10; in fixed point 11 and 12) at the edges of its shapes: radial sizes around a
warp's 16 or 32 elements, every band width, odd sizes, rows of no, one and up to nine terms, real and
complex bands, several time functions.  Reference: dense numpy in FP64."""
import numpy as np
import pytest

from pyprop_gb300 import _native

pytestmark = pytest.mark.gpu


def _operator(h, rng, nl, nr, kb):
    """Adds potentials to h; returns [(time function, rows, columns, dense radial matrices)]."""
    W = 2 * kb + 1
    out = []

    def add(storage, pairs, npairs, complex_band, td):
        data = np.zeros((npairs, W * nr), dtype=np.complex128)
        M = np.zeros((npairs, nr, nr), dtype=np.complex128)
        for q in range(npairs):
            for d in range(-kb, kb + 1):
                j = np.arange(max(0, -d), min(nr, nr - d))          # entry (j + d, j)
                v = rng.standard_normal(len(j)) + (1j * rng.standard_normal(len(j)) if complex_band else 0)
                M[q, j + d, j] = v
                data[q, j * W + kb + d] = v
        h.add_potential(storage, pairs, kb, data, td)
        if storage == _native.STORAGE_SIMP:
            rows, cols = pairs[:, 0], pairs[:, 1]
        else:
            rows = cols = np.arange(nl)
            M = np.broadcast_to(M, (nl, nr, nr))
        out.append((td, rows, cols, M))

    pairs = [(l, l - 1) for l in range(1, nl)] + [(l - 1, l) for l in range(1, nl)]
    if nl > 4:
        pairs += [(2, q) for q in range(nl)]                       # a long row; row nl - 1 loses its terms
        pairs = [p for p in pairs if p[0] != nl - 1]
    if pairs:
        add(_native.STORAGE_SIMP, np.array(pairs, dtype=np.int32), len(pairs), False, 1)
        add(_native.STORAGE_SIMP, np.array(pairs[:2], dtype=np.int32), len(pairs[:2]), True, 2)
    if nl <= 4:
        add(_native.STORAGE_DIAG, None, nl, True, 0)
        add(_native.STORAGE_IDENT, None, 1, False, 2)
    return out


SHAPES = [(1, 9, 6), (2, 15, 6), (3, 16, 6), (4, 17, 1), (5, 31, 2), (6, 32, 3), (7, 33, 4), (9, 47, 5), (5, 129, 7),
          (3, 300, 8)]


def _apply(nl, nr, kb, variant, precision, scale=1.0):
    """(result, exact, sum of |A| |x|, W max|A| max|x| of an element's row and whole vector, terms per row)."""
    import torch
    rng = np.random.default_rng(100 * nr + kb)
    h = _native.Handle(nl, nr, precision, 4, 0, False, 0)
    h.set_overlap(1, np.tile([0.0, 1.0], nr))
    ops = _operator(h, rng, nl, nr, kb)
    h.finalize()
    assert h.autotune(variant) == variant
    x = (rng.standard_normal((nl, nr)) + 1j * rng.standard_normal((nl, nr))) * scale
    src = torch.as_tensor(x).to("cuda", torch.complex128 if precision == _native.FP64 else torch.complex64)
    dst = torch.full_like(src, 7.0)
    scal = [1.0, 0.37, -1.9]
    h.matvec(src, dst, scal[1:], balanced=False)
    x = src.cpu().numpy().astype(np.complex128)
    want, size, peak, terms = np.zeros((nl, nr), complex), np.zeros((nl, nr)), np.zeros((nl, nr)), np.zeros((nl, 1))
    for td, rows, cols, M in ops:
        for r, c, A in zip(rows, cols, M):
            want[r] += scal[td] * (A @ x[c])
            size[r] += abs(scal[td]) * ((abs(A.real) + abs(A.imag)) @ (abs(x[c].real) + abs(x[c].imag)))
            peak[r] += abs(scal[td]) * 2 * (2 * kb + 1) * abs(A).max(axis=1) * abs(x[c]).max()
            terms[r] += 2
    return dst.cpu().numpy().astype(np.complex128), want, size, peak, terms


@pytest.mark.parametrize("nl,nr,kb", SHAPES)
@pytest.mark.parametrize("variant", [9, 10])
@pytest.mark.parametrize("precision", [_native.FP64, _native.FP32_MIXED])
def test_term_per_warp(nl, nr, kb, variant, precision):
    """Elementwise: FP64 rounds each of an element's products and sums once, 2^-53 of |A| |x| each; complex64 rounds the
    exact sum (coefficients and sums hold 2^-40 of |A| |x| at least)."""
    got, want, size, _, terms = _apply(nl, nr, kb, variant, precision)
    if precision == _native.FP64:
        bound = size * 2.0 ** -53 * (2 * (2 * kb + 1) + 4 * terms + 8)
    else:
        bound = 2.0 ** -24 * np.sqrt(2) * abs(want) + size * 2.0 ** -40
    assert (abs(got - want) <= bound).all()


@pytest.mark.parametrize("nl,nr,kb", SHAPES)
@pytest.mark.parametrize("variant", [11, 12])
@pytest.mark.parametrize("scale", [1.0, 1e-290, 1e290])
def test_fixed_point(nl, nr, kb, variant, scale):
    """Each factor is rounded to 2^-58 of the largest and the low digits' product dropped (2^-60), each product; the
    terms' sums round to 2^-53.  (numpy's own sums round as FP64's.)"""
    got, want, size, peak, terms = _apply(nl, nr, kb, variant, _native.FP64, scale)
    bound = peak * 3 * 2.0 ** -58 + size * 2.0 ** -53 * (2 * (2 * kb + 1) + 4 * terms + 8)
    assert (abs(got - want) <= bound).all()


@pytest.mark.parametrize("variant", [11, 12])
def test_fixed_point_nonfinite(variant):
    """An infinity or a NaN reaches every element whose sum reads it."""
    import torch
    nr = 100
    h = _native.Handle(1, nr, _native.FP64, 4, 0, False, 0)
    h.set_overlap(1, np.tile([0.0, 1.0], nr))
    h.add_potential(_native.STORAGE_DIAG, None, 2, np.ones((1, 5 * nr), dtype=np.complex128), False)
    h.finalize()
    h.autotune(variant)
    for bad in (float("inf"), float("nan")):
        src = torch.ones((1, nr), dtype=torch.complex128, device="cuda")
        src[0, 50] = complex(bad, 0.0)
        dst = torch.zeros_like(src)
        h.matvec(src, dst, 0.0, balanced=False)
        assert not bool(torch.isfinite(dst.real[0, 48:53]).any())
        assert bool((dst.real[0, 5:25] == 5.0).all()) and bool((dst.real[0, 75:95] == 5.0).all())
