"""The cooperative recursion around the sizes where it ends: one row, partial tiles, the last
size whose tiles are all resident and the next one, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-10, "dd": 1e-10, "mixed": 2e-5}      # the stated bounds


# 152 SMs x 4 FP64 CTAs x 256 / 8 lanes = 19,456 rows; the other types reach further or less
@pytest.mark.parametrize("n,R", [(1, 2), (3, 8), (31, 5), (257, 2), (4097, 6), (19456, 8), (19457, 8), (40000, 8)])
@pytest.mark.parametrize("precision", ["fp64", "dd", "mixed"])
@pytest.mark.parametrize("doubling", [True, False])
@pytest.mark.parametrize("varied", [False, True])
def test_matches_oracle(gpu, n, R, precision, doubling, varied):
    X = tb.PartialLattice(tb.Chain().add_hopping("A", "A", (1,), 0.3).add_hopping("A", "A", (7,), 0.1), (n,))
    X.set_scalar_values(np.linspace(-0.15, 0.15, n))
    H = X.get_Hamiltonian_sparse(float)
    cp, ri, v = H.to_csc()
    if varied:                                         # no row classes once rows outnumber them
        rows = np.repeat(np.arange(n), np.diff(cp))
        v = v * (1 - 0.2 * np.cos(ri * 0.37) * np.cos(rows * 0.37))
    A = tb.SparseMatrix.from_csc(n, n, cp, ri, v)
    M = 21
    kets = orc.random_phase_kets(n, R, 1)
    bras = kets if doubling else orc.random_phase_kets(n, R, 2)
    S = tb.KpmSolver(A, R, precision, doubling)
    mu = S.run(M, bras, kets)
    assert np.array_equal(mu, S.run(M, bras, kets)) and np.array_equal(mu, S.run(M, bras, kets))
    assert np.max(np.abs(mu - orc.cheb_moments(n, cp, ri, v, M, bras, kets))) <= TOL[precision] * R
