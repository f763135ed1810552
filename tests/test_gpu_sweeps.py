"""Steps that sweep vectors past L2 in alternating directions: the same values as those of
the same vectors a few at a time, which stay in L2 and are swept one way."""
import numpy as np
import pytest

import tight_binding_gb300 as tb
from tight_binding_gb300.serving import model_bounds, model_cell

pytestmark = pytest.mark.gpu


def _matrix(kind, n):
    X = tb.PartialLattice(model_cell(kind), n)
    X.set_scalar_values(np.random.default_rng(4).random(X.get_total_number()) - 0.5)
    H = X.get_Hamiltonian_periodic_extend_bare_sparse([1] * len(n))
    return tb.GreenFunction(16, H, *model_bounds(kind, 1.0))


@pytest.mark.parametrize("precision,eps", [("dd", 2.0 ** -45), ("fp64", 2.0 ** -52), ("mixed", 2.0 ** -23)])
@pytest.mark.parametrize("n", [(401, 317)])
def test_expansion(precision, eps, n):
    """12 vectors of 254,234 sites: 3 blocks of 49 MB (complex64: 24 MB each, 73 MB).  A row's
    value is the same few operations either way: at most 9 roundings a term and row, whose
    growth over the 30 terms (|U_k| <= k + 1) stays within 9 * 30 * 31 / 2."""
    G = _matrix("honeycomb", n)
    kets = tb.bases_of_uniform_ampl_with_random_phases(G.scaled_HE.shape[0], 12, 3)
    coef = np.random.default_rng(1).normal(size=30) + 0.5j
    whole = tb.cheb_expand(G.scaled_HE, coef, kets, precision)
    parts = np.hstack([tb.cheb_expand(G.scaled_HE, coef, kets[:, r:r + 2], precision) for r in range(0, 12, 2)])
    assert np.abs(whole - parts).max() <= 9 * 30 * 31 / 2 * eps * np.abs(coef).max() * np.abs(kets).max()


@pytest.mark.parametrize("form", [{"fuse_ops": True}, {"fuse_ops": True, "both_sides": True}])
def test_kubo_opt_in_forms(form):
    """8 vectors of 254,234 sites, as many tiles as make the steps' CTAs wide: the opt-in forms
    store the same bits, whichever the number of threads per CTA (the budget holds chunks of
    four vectors, 195 MB, in every form)."""
    G = _matrix("honeycomb", (401, 317))
    X = tb.PartialLattice(model_cell("honeycomb"), (401, 317))
    v = tb.commutator(G.scaled_HE, X.op_position(0))
    plain = tb.kubo_mu(G.scaled_HE, v, None, None, v, M=12, R=8, seed=3, budget_gb=0.2)
    chunks = tb.kubo_last_timing()["chunks"]
    assert np.array_equal(tb.kubo_mu(G.scaled_HE, v, None, None, v, M=12, R=8, seed=3, budget_gb=0.2, **form), plain)
    assert chunks == tb.kubo_last_timing()["chunks"] == 2
    tb.kubo_release()


@pytest.mark.parametrize("operator", [False, True])
def test_kubo_blocks(operator):
    """Double-float recursions of 16 vectors of 64^3 sites in chunks of four, two blocks of 17 MB,
    against two vectors at a time.  Sums of 64 FP32 products of norm-one vectors' entries on
    either side."""
    G = _matrix("fcc", (64, 64, 64))
    n = G.scaled_HE.shape[0]
    X = tb.PartialLattice(model_cell("fcc"), (64, 64, 64))
    v = tb.commutator(G.scaled_HE, X.op_position(0)) if operator else None
    kets = tb.bases_of_uniform_ampl_with_random_phases(n, 16, 5)
    mu = lambda k: tb.kubo_mu(G.scaled_HE, v, None, None, None, M=12, kets=k, recursion="dd")
    whole = mu(kets)
    assert tb.kubo_last_timing()["chunks"] == 4
    parts = sum(mu(kets[:, r:r + 2]) for r in range(0, 16, 2))
    size = 16.0
    if operator:                                         # the largest column sum of |v|, which bounds |v x|
        p, _, a = v.to_csc()
        size *= np.add.reduceat(np.abs(a), np.minimum(p[:-1], len(a) - 1)).max()
    assert np.abs(whole - parts).max() <= 2 * np.sqrt(2) * 64 * 2.0 ** -24 * size
    tb.kubo_release()
