"""The cooperative recursion's give-up path: with a limit of no further polls its CTAs leave at
the first meeting that others have not reached, the call reports it, and the plan's next run
with the default limit is right."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
import tight_binding_gb300 as tb
from tight_binding_gb300 import capi

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-10, "dd": 1e-10, "mixed": 2e-5}      # the stated bounds


@pytest.mark.parametrize("precision", ["fp64", "dd", "mixed"])
@pytest.mark.parametrize("doubling", [True, False])
@pytest.mark.parametrize("varied", [False, True])      # row classes, ELL
def test_gives_up_and_recovers(gpu, precision, doubling, varied):
    X = tb.PartialLattice(tb.Square().add_hopping("A", 1, 0.24), (61, 50))
    A = X.get_Hamiltonian_periodic_extend_bare_sparse([1, 1], float)
    if varied:
        cp, ri, v = A.to_csc()
        rows = np.repeat(np.arange(A.shape[0]), np.diff(cp))
        A = tb.SparseMatrix.from_csc(*A.shape, cp, ri, v * (1 - 0.2 * np.cos(ri * 0.37) * np.cos(rows * 0.37)))
    assert (A.row_classes() == 0) == varied
    cp, ri, v = A.to_csc()
    n, R, M = A.shape[0], 8, 40
    kets = orc.random_phase_kets(n, R, 1)
    bras = kets if doubling else orc.random_phase_kets(n, R, 2)
    S = tb.KpmSolver(A, R, precision, doubling)
    try:
        capi.check(capi.lib().tbk_set_wait_limit(0))
        with pytest.raises(tb.TbkError) as e:
            S.run(M, bras, kets)
        assert e.value.code == capi.TBK_ERR_TIMEOUT
    finally:
        capi.check(capi.lib().tbk_set_wait_limit(-1))
    mu = S.run(M, bras, kets)
    assert np.max(np.abs(mu - orc.cheb_moments(n, cp, ri, v, M, bras, kets))) <= TOL[precision] * R
