"""Bound states at the edges of the kernels' shapes: radial sizes around the 32-row blocks of the
sweeps and down to the band width, band widths 3 to 8, upper ends on both sides of zero (intervals of
more than 2^63 doubles), more states than are asked for.  Reference: numpy's dense eigenvalues of
U^-T H U^-1."""
import numpy as np
import pytest

from pyprop_gb300 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,order", [(8, 7), (31, 4), (32, 5), (33, 7), (64, 6), (65, 8), (96, 9), (129, 7), (300, 7)])
@pytest.mark.parametrize("emax", [-0.05, 0.0, 12.0])
def test_eigenpairs(nr, order, emax):
    import torch
    from pyprop_gb300.batch import HydrogenProblem
    from pyprop_gb300.observables import _dense_from_diagonals, _symmetric_bands
    p = HydrogenProblem(lmax=2, nr=nr, rmax=0.3 * nr, order=order, m=4)
    S = _dense_from_diagonals(p.Sdiag, p.kd, nr)
    Hb = np.stack([_symmetric_bands(p.static[l], nr, p.kb) for l in range(3)])
    most = 12
    counts, energies, vecs = _native.bound_states(torch.as_tensor(Hb).cuda(), torch.as_tensor(p.Sdiag).cuda(), emax, most)
    vecs = vecs.cpu().numpy()
    Li = np.linalg.inv(np.linalg.cholesky(S))
    for l in range(3):
        H = _dense_from_diagonals(Hb[l], p.kd, nr)
        e = np.linalg.eigvalsh(Li @ H @ Li.T)
        want = e[e < emax]
        assert counts[l] == len(want)
        k = min(most, len(want))
        # numpy's own error is a few roundings of the largest eigenvalue
        tol = 1e-12 + 1e-15 * nr * np.abs(e).max()
        assert np.max(np.abs(energies[l, :k] - want[:k]), initial=0.0) < tol
        assert not energies[l, k:].any() and not vecs[l, k:].any()
        for j in range(k):
            v = vecs[l, j]
            assert abs(v @ S @ v - 1.0) < 1e-12
            assert np.linalg.norm(H @ v - energies[l, j] * (S @ v)) < tol * np.linalg.norm(v)
