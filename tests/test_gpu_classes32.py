"""Row classes of FP32 values (rational fluxes, commutators) and joint classes of H~ and
an operator: complex64 results against the ELL form of the same matrices, bit for bit."""
from __future__ import annotations

import os

import numpy as np
import pytest

import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu


def _system(kind, span, flux):
    cell = {"square": tb.Square, "honeycomb": tb.Honeycomb, "fcc": tb.FCC}[kind]().add_hopping("A", 1, 1.0)
    X = tb.PartialLattice(cell, span)
    X.set_scalar_values(np.random.default_rng(2).random(X.get_total_number()) - 0.5)
    if flux:
        G = np.zeros((3, 3))
        G[1, 0] = 2 * np.pi / flux
        X.set_gauge_linear(G)
    per = [0 if flux else 1] + [1] * (len(span) - 1)
    H = X.get_Hamiltonian_periodic_extend_bare_sparse(per, complex if flux else float)
    A = tb.GreenFunction(2, H, -13.0, 13.0).scaled_HE
    return A, tb.commutator(A, X.op_position(0))


def _ell(build):
    os.environ["TBK_NO_CLASSES"] = "1"
    try:
        return build()
    finally:
        del os.environ["TBK_NO_CLASSES"]


SYSTEMS = [("square", (70, 33), 16), ("honeycomb", (31, 29), 0), ("fcc", (9, 8, 7), 0), ("square", (300, 12), 0)]


@pytest.mark.parametrize("kind,span,flux", SYSTEMS)
def test_expansion_equals_ell(gpu, kind, span, flux):
    A, v = _system(kind, span, flux)
    kets = tb.bases_of_uniform_ampl_with_random_phases(A.shape[0], 6, 1)
    c = [0.2, 0.5j, -0.3, 0.1]
    for B in (A, v):
        got = tb.cheb_expand(B, c, kets, "mixed")

        def forced():
            cp, ri, x = B.to_csc()
            return tb.cheb_expand(tb.SparseMatrix.from_csc(*B.shape, cp, ri, x), c, kets, "mixed")

        assert np.array_equal(got, _ell(forced))


# 1, 2, 3 vectors (one lane, two, padded), a run-time width, both stores
@pytest.mark.parametrize("tensor", [False, True])
@pytest.mark.parametrize("R", [1, 2, 3, 6])
@pytest.mark.parametrize("kind,span,flux", SYSTEMS)
def test_kubo_equals_ell(gpu, kind, span, flux, R, tensor):
    M = 9

    def solve():
        A, v = _system(kind, span, flux)
        return (tb.kubo_mu(A, None, None, v, v, M, R, seed=2, tensor=tensor),
                tb.kubo_mu(A, v, v, None, None, M, R, seed=2, tensor=tensor))

    for a, b in zip(solve(), _ell(solve)):
        assert np.array_equal(a, b)
