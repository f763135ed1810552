"""Vector counts whose chunk width has no instantiation of its own (odd, between powers
of two, over one chunk's cap), in every precision and matrix form, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-10, "dd": 1e-10, "mixed": 2e-5}      # the stated bounds, relative to mu_0


def _matrix(form):
    cell = tb.Honeycomb().add_hopping("A", 1, 1.0)
    X = tb.PartialLattice(cell, (9, 11))                # 198 sites: a partial slice and partial tiles
    X.set_scalar_values(np.random.default_rng(5).random(X.get_total_number()) - 0.5)
    if form == "flux":
        G = np.zeros((3, 3))
        G[1, 0] = 0.21
        X.set_gauge_linear(G)
        H = X.get_Hamiltonian_sparse(complex)
    else:
        H = X.get_Hamiltonian_periodic_extend_bare_sparse([1, 1], float)
    A = tb.GreenFunction(2, H, -3.4, 3.4).scaled_HE
    if form != "ell":
        return A
    cp, ri, v = A.to_csc()                              # every row its own values: more than 255 classes
    n = len(cp) - 1
    w = np.random.default_rng(6).uniform(0.8, 1.0, 2 * n)
    cols = [(ri[cp[j]:cp[j + 1]] + b * n, v[cp[j]:cp[j + 1]]) for b in (0, 1) for j in range(n)]
    vals = [x * w[r] * w[q] for q, (r, x) in enumerate(cols)]
    cp2 = np.concatenate([[0], np.cumsum([len(r) for r, _ in cols])])
    return tb.SparseMatrix.from_csc(2 * n, 2 * n, cp2, np.concatenate([r for r, _ in cols]), np.concatenate(vals))


@pytest.mark.parametrize("doubling", [True, False])
@pytest.mark.parametrize("precision", ["mixed", "dd", "fp64"])
@pytest.mark.parametrize("form", ["classes", "ell", "flux"])
@pytest.mark.parametrize("R", [3, 5, 9, 20, 31, 33, 50, 67])
def test_moments(gpu, R, form, precision, doubling):
    A = _matrix(form)
    assert (A.row_classes() > 0) == (form != "ell")
    cp, ri, v = A.to_csc()
    n, M = A.shape[0], 24
    kets = orc.random_phase_kets(n, R, 1)
    bras = kets if doubling else orc.random_phase_kets(n, R, 2)
    mu = tb.KpmSolver(A, R, precision, doubling).run(M, bras, kets)
    ref = orc.cheb_moments(n, cp, ri, v, M, bras, kets)
    # bras other than kets: relative to the R unit norms, as mu_0 is for bras == kets
    assert np.max(np.abs(mu - ref)) <= TOL[precision] * R


@pytest.mark.parametrize("precision", ["mixed", "dd", "fp64"])
@pytest.mark.parametrize("R", [3, 7, 18, 37])
def test_expansion_and_view(gpu, R, precision):
    A = _matrix("ell")
    D = np.zeros(A.shape)
    cp, ri, v = A.to_csc()
    for j in range(A.shape[0]):
        D[ri[cp[j]:cp[j + 1]], j] = v[cp[j]:cp[j + 1]]
    kets = orc.random_phase_kets(A.shape[0], R, 3)
    c = np.array([0.3, -0.2j, 0.5, 0.1 + 0.4j])
    T = [kets, D @ kets]
    T += [2 * D @ T[1] - T[0]]
    T += [2 * D @ T[2] - T[1]]
    tol = TOL[precision] * np.max(np.abs(kets)) * 4
    assert np.max(np.abs(tb.cheb_expand(A, c, kets, precision) - sum(a * t for a, t in zip(c, T)))) <= tol
    for got, want in zip(tb.Cheb_first_kind_seq_on_bases(A, 4, kets, precision), T):
        assert np.max(np.abs(got - want)) <= tol


@pytest.mark.parametrize("tensor", [False, True])
@pytest.mark.parametrize("recursion", ["mixed", "dd", "fp64"])
@pytest.mark.parametrize("R", [3, 5, 9])
def test_kubo(gpu, R, recursion, tensor):
    A = _matrix("classes")
    n, M = A.shape[0], 20
    X = tb.SparseMatrix.from_csc(n, n, np.arange(n + 1), np.arange(n), np.arange(n) * 0.01)
    va = tb.commutator(A, X)
    mu = tb.kubo_mu(A, va, va, None, None, M, R, seed=4, tensor=tensor, recursion=recursion)
    ref = tb.kubo_mu(A, va, va, None, None, M, R, seed=4, recursion="fp64", fp64_blocks=True)
    assert np.max(np.abs(mu - ref)) <= 2e-5 * np.max(np.abs(ref))
    one = sum(tb.kubo_mu(A, va, va, None, None, M, kets=k[:, None], recursion="fp64", fp64_blocks=True)
              for k in orc.random_phase_kets(n, R, 4).T)
    assert np.max(np.abs(ref - one)) <= 1e-10 * np.max(np.abs(ref))
