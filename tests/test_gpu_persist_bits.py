"""The cooperative recursion gives the bits of the per-step launches, at numbers of CTAs that
are no power of two and beyond one partial sum per thread of the reduction (256, 512)."""
from __future__ import annotations

import numpy as np
import pytest

import tight_binding_gb300 as tb
from tight_binding_gb300 import capi

pytestmark = pytest.mark.gpu


# at R = 8 a CTA has 32 rows in FP64, 64 in the other precisions
@pytest.mark.parametrize("n", [70, 3100, 8200, 16500, 19456, 33000])
@pytest.mark.parametrize("precision", ["fp64", "dd", "mixed"])
@pytest.mark.parametrize("doubling", [True, False])
@pytest.mark.parametrize("varied", [False, True])      # row classes, ELL
@pytest.mark.parametrize("zigzag", [True, False])
def test_equals_steps(gpu, n, precision, doubling, varied, zigzag):
    X = tb.PartialLattice(tb.Chain().add_hopping("A", "A", (1,), 0.3).add_hopping("A", "A", (7,), 0.1), (n,))
    X.set_scalar_values(np.linspace(-0.15, 0.15, n))
    cp, ri, v = X.get_Hamiltonian_sparse(float).to_csc()
    if varied:
        rows = np.repeat(np.arange(n), np.diff(cp))
        v = v * (1 - 0.2 * np.cos(ri * 0.37) * np.cos(rows * 0.37))
    A = tb.SparseMatrix.from_csc(n, n, cp, ri, v)
    kets = tb.bases_of_uniform_ampl_with_random_phases(n, 8, 1)
    bras = kets if doubling else tb.bases_of_uniform_ampl_with_random_phases(n, 8, 2)
    base = 0 if zigzag else capi.FLAG_NO_L2_ZIGZAG

    def mu(flags):
        return tb.KpmSolver(A, 8, precision, doubling, base | flags).run(30, bras, kets)

    assert np.array_equal(mu(0), mu(capi.FLAG_NO_GRAPH))
    if precision != "mixed":                           # two-step passes are complex64 only: per-step launches
        assert np.array_equal(mu(0), mu(capi.FLAG_TWO_STEP))
