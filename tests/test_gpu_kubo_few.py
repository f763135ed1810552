"""kubo_mu around the numbers of steps from which it uses a second stream (8) and takes the
operators' products inside the recursion (32): the same bits with the product asked for, and
the complex128 blocks' values."""
from __future__ import annotations

import numpy as np
import pytest

import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,R,budget", [(1, 2, 0.0), (2, 3, 0.0), (7, 2, 0.0), (8, 2, 0.0), (31, 2, 0.0), (32, 2, 0.0),
                                        (4, 8, 6e-5), (16, 4, 2e-4)])       # chunks of 2
@pytest.mark.parametrize("which", ["bastin", "greenwood", "plain"])
@pytest.mark.parametrize("tensor", [True, False])
@pytest.mark.parametrize("flux", [0, 16])
def test_forms(gpu, M, R, budget, which, tensor, flux):
    X = tb.PartialLattice(tb.Square().add_hopping("A", 1, 1.0), (20, 16))
    X.set_scalar_values(np.random.default_rng(1).random(320) - 0.5)
    if flux:
        K = np.zeros((3, 3))
        K[1, 0] = 2 * np.pi / flux
        X.set_gauge_linear(K)
    H = X.get_Hamiltonian_periodic_extend_bare_sparse([0 if flux else 1, 1], complex if flux else float)
    A = tb.GreenFunction(2, H, -5.0, 5.0).scaled_HE
    v, u = (tb.commutator(A, X.op_position(k)) for k in range(2))
    ops = {"bastin": (None, None, v, u), "greenwood": (v, v, None, None), "plain": (None,) * 4}[which]
    mu = tb.kubo_mu(A, *ops, M=M, R=R, seed=2, tensor=tensor, budget_gb=budget)
    assert tb.kubo_last_timing()["chunks"] == (1 if not budget else R // 2)
    assert np.array_equal(mu, tb.kubo_mu(A, *ops, M=M, R=R, seed=2, tensor=tensor, budget_gb=budget, fuse_ops=True))
    ref = tb.kubo_mu(A, *ops, M=M, R=R, seed=2, fp64_blocks=True)
    assert np.max(np.abs(mu - ref)) <= 2e-5 * np.max(np.abs(ref))
