"""Gram-Schmidt at the edges of its grid: sizes around a warp's chunk, one CTA per SM, odd sizes, chunks
that fit in shared memory or not, with and without re-orthogonalisation.  Reference: the Hessenberg
matrix of a diagonal operator by numpy with full re-orthogonalisation."""
import numpy as np
import pytest

from pyprop_gb300 import _native

pytestmark = pytest.mark.gpu


def _handle(nl, nr, m, dorth, diag, precision=_native.FP64):
    """A diagonal operator in an orthonormal basis (overlap factor 1, bandwidth 1)."""
    one = np.zeros((nl, 3 * nr), dtype=np.complex128)
    one[:, np.arange(nr) * 3 + 1] = diag.reshape(nl, nr)
    band = np.zeros((nr, 2))
    band[:, 1] = 1.0
    h = _native.Handle(nl, nr, precision, m, 0, dorth, 0)
    h.set_overlap(1, band)
    h.add_potential(_native.STORAGE_DIAG, None, 1, one, False)
    h.finalize()
    return h


def _arnoldi(diag, x, m):
    """The Hessenberg matrix (m x m, betas below the diagonal) with full re-orthogonalisation."""
    a, v = diag, x
    V = [v / np.sqrt(np.sum(np.abs(v) ** 2))]
    H = np.zeros((m, m), dtype=np.complex128)
    for J in range(m):
        w = a * V[J]
        for _ in range(2):
            for k in range(J + 1):
                c = np.sum(V[k].conj() * w)
                H[k, J] += c
                w = w - c * V[k]
        beta = np.sqrt(np.sum(np.abs(w) ** 2))
        if J + 1 < m:
            H[J + 1, J] = beta
            V.append(w / beta)
    return H


SHAPES = [(1, 9, 4), (1, 31, 5), (4, 8, 5), (3, 11, 5), (5, 52, 16), (16, 304, 17), (16, 304, 45), (9, 541, 20),
          (17, 1001, 33), (64, 1500, 24)]


@pytest.mark.parametrize("nl,nr,m", SHAPES)
@pytest.mark.parametrize("dorth", [False, True])
def test_hessenberg(nl, nr, m, dorth):
    """A spectrum spread over [-1, 1]: every beta is near 1/2, so nothing amplifies the rounding of the
    sums: m vectors of at most log2(N) + m roundings of 2^-53 each."""
    import torch
    rng = np.random.default_rng(nl * nr + m)
    N = nl * nr
    diag = rng.permutation(np.linspace(-1.0, 1.0, N))
    x = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    want = _arnoldi(diag, x, m)
    assert np.abs(np.diag(want, -1)).min() > 0.2
    h = _handle(nl, nr, m, dorth, diag)
    d = torch.as_tensor(x.reshape(nl, nr)).cuda()
    h.advance(d, np.zeros(1), 0.01)
    got = 1j * h.hessenberg() / 0.01                   # the exponential leaves -i dt H
    assert np.abs(got - want).max() < m * (np.log2(N) + m) * 2.0 ** -53


@pytest.mark.parametrize("c", [1.01, 1.3, 1.5, 1.7, 1.9, 1.99, 222.0, 255.0, 288.8, 300.0])
@pytest.mark.parametrize("dorth", [False, True])
def test_equal_partial_sums(c, dorth):
    """A uniform vector and +-c alternating: every CTA's partial sum is the same, whatever its mantissa.  Each element goes
    through fewer than 16 roundings."""
    import torch
    nl, nr = 16, 304
    h = _handle(nl, nr, 2, dorth, c * (-1.0) ** np.arange(nl * nr))
    d = torch.full((nl, nr), 0.6 + 0.8j, dtype=torch.complex128, device="cuda")
    h.advance(d, np.zeros(1), 0.01)
    want = c * np.array([[0.0, 1.0], [1.0, 0.0]])
    assert np.abs(1j * h.hessenberg() / 0.01 - want).max() < 2.0 ** -49 * c
