"""Spectral ranges of matrices whose entries are far from 1 (energies in odd units)."""
from __future__ import annotations

import numpy as np
import pytest

import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu


# powers of two: the same recursion but for the exponents.  The residuals and the Sturm sequence
# square the scalars, so 1e150 is near the end of the range.  (Small entries are another matter:
# the bisection's and the breakdown's thresholds are absolute below 1.)
@pytest.mark.parametrize("exponent", [490, 400, 345, 199, 60])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("vacancy", [False, True])
def test_power_of_two(gpu, exponent, cplx, vacancy):
    X = tb.PartialLattice(tb.Square().add_hopping("A", "A", (1, 0), 0.6 + 0.8j if cplx else 1.0)
                          .add_hopping("A", "A", (0, 1), 0.7), (40, 31))
    X.set_scalar_values(np.random.default_rng(0).random(40 * 31) - 0.5)
    if vacancy:
        X.remove_atoms("A", [[3, 4]])
    H = X.get_Hamiltonian_sparse(complex if cplx else float)
    n, (cp, ri, v) = H.shape[0], H.to_csc()
    ref = np.array(tb.spectral_range(H, iters=150, seed=3))
    assert ref[0] < -2 and ref[1] > 2
    f = 2.0 ** exponent
    got = np.array(tb.spectral_range(tb.SparseMatrix.from_csc(n, n, cp, ri, v * f), iters=150, seed=3))
    # the bisection stops at 1e-15 of the interval; the residuals of converged vectors are rounding,
    # so they are only bounded
    assert np.all(np.abs(got[:2] / f - ref[:2]) <= 1e-14 * np.abs(ref[:2]))
    assert np.all(np.isfinite(got)) and np.all(got[2:] / f <= np.maximum(ref[2:], 1e-6) * 10)


def test_zero_and_not_finite(gpu):
    n = 50
    cp, ri = np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32)
    assert np.allclose(tb.spectral_range(tb.SparseMatrix.from_csc(n, n, cp, ri, np.zeros(n)))[:2], 0)
    v = np.ones(n)
    v[7] = np.nan
    assert not np.all(np.isfinite(tb.spectral_range(tb.SparseMatrix.from_csc(n, n, cp, ri, v))))
