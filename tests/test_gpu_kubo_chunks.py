"""The chunk width of a Kubo solve whose stores no pool keeps: narrower than R, the same
moment matrix as the widths that a budget forces."""
import numpy as np
import pytest

import tight_binding_gb300 as tb
from tight_binding_gb300.serving import model_bounds, model_cell

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,budgets,chunks", [(8, (0.0, 18.0, 4.5), [2, 2, 4]), (5, (0.0, 10.0), [1, 2])])
def test_widths(R, budgets, chunks):
    """64^3 sites x 512 blocks x 2 sides x 8 bytes: 2.15 GB a vector; 8 vectors are past the 16
    GiB that are kept.  Each width sums the same products in other groups of 128, each 24
    additions in FP32: at most 24 x 2^-23 of the largest entry on either side, 6e-6."""
    n, M = (64, 64, 64), 512
    X = tb.PartialLattice(model_cell("fcc"), n)
    X.set_scalar_values(np.random.default_rng(4).random(64 ** 3) - 0.5)
    H = X.get_Hamiltonian_periodic_extend_bare_sparse([1, 1, 1])
    G = tb.GreenFunction(M, H, *model_bounds("fcc", 1.0))
    v = tb.commutator(G.scaled_HE, X.op_position(0))
    out, seen = [], []
    for b in budgets:
        out.append(tb.kubo_mu(G.scaled_HE, v, v, M=M, R=R, seed=2, tensor=True, budget_gb=b))
        seen.append(tb.kubo_last_timing()["chunks"])
    assert seen == chunks
    for o in out[1:]:
        assert np.abs(o - out[0]).max() <= 6e-6 * np.abs(out[0]).max()
    tb.kubo_release()
