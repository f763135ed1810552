"""The Lanczos kernels in their four forms (real / complex H, row classes / ELL) at
sizes around one CTA and one slice, against dense eigenvalues."""
from __future__ import annotations

import numpy as np
import pytest

import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vacancy", [False, True])
@pytest.mark.parametrize("t", [1.0, 0.6 + 0.8j])
@pytest.mark.parametrize("span", [(1, 2), (4, 8), (5, 51), (16, 16), (1, 257), (24, 43)])
def test_forms_match_dense(gpu, span, t, vacancy):
    cell = tb.Square().add_hopping("A", "A", (1, 0), t).add_hopping("A", "A", (0, 1), 0.7 * t)
    X = tb.PartialLattice(cell, span)
    n = X.get_total_number()
    X.set_scalar_values(np.random.default_rng(n).random(n) - 0.5)
    if vacancy:
        X.remove_atoms("A", [[0, span[1] // 2]])
    H = X.get_Hamiltonian_sparse(complex if isinstance(t, complex) else float)
    cp, ri, v = H.to_csc()
    D = np.zeros((n, n), dtype=complex)
    for j in range(n):
        D[ri[cp[j]:cp[j + 1]], j] = v[cp[j]:cp[j + 1]]
    w = np.linalg.eigvalsh(D)
    e0, e1, _, _ = tb.spectral_range(H, iters=400, seed=3)
    # 400 steps converge the extremes of these sizes to rounding of the recursion
    tol = 1e-10 * max(abs(w[0]), abs(w[-1]), 1.0)
    assert abs(e0 - w[0]) <= tol and abs(e1 - w[-1]) <= tol
