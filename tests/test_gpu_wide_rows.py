"""Double-float class-form steps of rows with more than 8 entries, which have kernels of their own
from 16 vectors on, against the oracle; shorter rows and fewer vectors beside them."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [8, 16, 20, 32, 48])
@pytest.mark.parametrize("doubling", [True, False])
@pytest.mark.parametrize("cell,span", [("fcc", (9, 8, 7)), ("fcc", (41, 40, 30)), ("square", (33, 21))])
def test_matches_oracle(gpu, cell, span, doubling, R):
    # first neighbours: 12 entries a row; second ones too on the square lattice: 8
    if cell == "fcc":
        X = tb.PartialLattice(tb.FCC().add_hopping("A", 1, 0.07), span)
    else:
        X = tb.PartialLattice(tb.Square().add_hopping("A", 1, 0.15).add_hopping("A", 2, 0.07), span)
    n = X.get_total_number()
    X.set_scalar_values(0.1 * (np.random.default_rng(1).random(n) - 0.5))
    A = X.get_Hamiltonian_periodic_extend_bare_sparse([1] * X.dim, float)
    assert A.row_classes() > 0
    cp, ri, v = A.to_csc()
    M = 17
    kets = orc.random_phase_kets(n, R, 1)
    bras = kets if doubling else orc.random_phase_kets(n, R, 2)
    mu = tb.KpmSolver(A, R, "dd", doubling).run(M, bras, kets)
    assert np.max(np.abs(mu - orc.cheb_moments(n, cp, ri, v, M, bras, kets))) <= 1e-10 * R
