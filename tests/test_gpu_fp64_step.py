"""The FP64 recursion step's two group forms (groups of four entries, single entries)
for rows of 0 to 8 neighbours, in the class form and the ELL form, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu


def _banded(n, reach, cplx, varied):
    """Hermitian band matrix (CSC): constant values (row classes) or its own in every row (ELL)."""
    rng = np.random.default_rng(reach)
    A = np.zeros((n, n), dtype=complex if cplx else float)
    for d in range(1, reach + 1):
        v = rng.uniform(0.05, 0.08, n - d) if varied else np.full(n - d, 0.07)
        if cplx:
            v = v * np.exp(0.3j * d)
        A += np.diag(v, d) + np.diag(np.conj(v), -d)
    A += np.diag(np.linspace(-0.3, 0.3, n))
    ri = [np.nonzero(A[:, j])[0] for j in range(n)]
    cp = np.concatenate([[0], np.cumsum([len(r) for r in ri])])
    return cp.astype(np.int32), np.concatenate(ri).astype(np.int32), np.concatenate([A[r, j] for j, r in enumerate(ri)])


@pytest.mark.parametrize("doubling", [True, False])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("varied", [False, True])
@pytest.mark.parametrize("reach", [0, 1, 2, 3, 4])
def test_row_widths_match_oracle(gpu, reach, varied, cplx, doubling):
    n, R, M = 300, 3, 40
    cp, ri, v = _banded(n, reach, cplx, varied)
    H = tb.SparseMatrix.from_csc(n, n, cp, ri, v)
    assert (H.row_classes() == 0) == (varied and reach > 0)
    kets = orc.random_phase_kets(n, R, 1)
    bras = kets if doubling else orc.random_phase_kets(n, R, 2)
    mu = tb.KpmSolver(H, R, "fp64", doubling).run(M, bras, kets)
    # the stated FP64 bound of the moments: 1e-10 of the R vectors' squared norms
    assert np.max(np.abs(mu - orc.cheb_moments(n, cp, ri, v, M, bras, kets))) <= 1e-10 * R


@pytest.mark.parametrize("h", [0.0, 5e-324, -2.0 ** -1023, -0.75, 2.0 ** 500])
def test_doubled_value_is_exact(gpu, h):
    A = tb.SparseMatrix.from_csc(1, 1, [0, 1], [0], np.array([h]))
    one = np.ones((1, 1))
    mu = tb.KpmSolver(A, 1, "fp64", False).run(3, one, one.copy())
    assert mu[1] == h and mu[2] == 2 * h * h - 1
