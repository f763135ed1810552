"""Moments of equal bras and kets where the matrix is not Hermitian, and the check that decides."""
from __future__ import annotations

import numpy as np
import pytest

import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu


def _csc(D, keep=None):
    """D column by column; keep: the stored pattern (default: the entries that are not zero)."""
    keep = D != 0 if keep is None else keep
    cols = [np.flatnonzero(keep[:, j]) for j in range(len(D))]
    cp = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    v = np.concatenate([D[c, j] for j, c in enumerate(cols)])
    return tb.SparseMatrix.from_csc(*D.shape, cp, np.concatenate(cols).astype(np.int32), v)


def _moments(D, kets, M):
    v0, v1 = kets, D @ kets
    mu = [np.vdot(kets, v0).real, np.vdot(kets, v1).real]
    for _ in range(2, M):
        v0, v1 = v1, 2 * (D @ v1) - v0
        mu.append(np.vdot(kets, v1).real)
    return np.array(mu)


def _skew(n=90):
    return np.diag(np.full(n - 1, 0.35), 1) + np.diag(np.full(n - 1, 0.25), -1)


def _gain_and_loss(n=90):
    return np.diag(np.full(n - 1, 0.3), 1) + np.diag(np.full(n - 1, 0.3), -1) + 0.05j * np.diag((-1.0) ** np.arange(n))


# bounds -1, 1: the rescale is the identity; the recursion's rounding as in the other moment tests
@pytest.mark.parametrize("D", [_skew(), _gain_and_loss()])
@pytest.mark.parametrize("precision", ["fp64", "dd"])
def test_moments_of_equal_bras_and_kets(gpu, precision, D):
    M, R = 24, 3
    G = tb.GreenFunction(M, _csc(D), -1.0, 1.0)
    kets = tb.bases_of_uniform_ampl_with_random_phases(len(D), R, 5)
    ref = _moments(D, kets, M)
    assert np.max(np.abs(G.imag(kets, kets, precision).moments - ref)) <= 1e-10 * R
    dos = tb.density_of_states_function(G, R, 5, precision)
    f = G.imag(kets, kets.copy(), precision)                   # bras that are not the kets: no product rule
    E = np.linspace(-0.7, 0.7, 9)
    assert np.max(np.abs(dos(E) + f(E) / (R * np.pi))) <= 1e-9


def test_is_hermitian(gpu):
    rng = np.random.default_rng(0)
    A = rng.normal(size=(70, 70)) + 1j * rng.normal(size=(70, 70))
    A = np.where(rng.random((70, 70)) < 0.1, A, 0)
    H = A + A.conj().T
    i, j = (int(k[0]) for k in np.nonzero(np.triu(H, 1)))

    def changed(at, value):
        B = H.copy()
        B[at] = value
        return B

    assert _csc(H).is_hermitian() and _csc(H.real.copy()).is_hermitian()
    assert _csc(changed((i, j), H[i, j] * (1 + 2.0 ** -51))).is_hermitian()
    assert not _csc(changed((i, j), H[i, j] * (1 + 2.0 ** -48))).is_hermitian()
    assert not _csc(changed((i, j), H[i, j].conj())).is_hermitian()
    assert not _csc(changed((i, j), 0)).is_hermitian()          # no mirror image
    assert not _csc(changed((i, j), np.nan)).is_hermitian()
    assert not _csc(changed((i, i), 1 + 1e-9j)).is_hermitian()
    keep = H != 0
    a, b = (int(k[0]) for k in np.nonzero(~keep & ~np.eye(70, dtype=bool)))
    keep[a, b] = True                                          # a stored zero needs none
    assert _csc(H, keep).is_hermitian()
    unsorted = tb.SparseMatrix.from_csc(2, 2, np.array([0, 2, 4], np.int32), np.array([1, 0, 0, 1], np.int32),
                                        np.array([0.5, 0.0, 0.5, 0.0]))
    assert not unsorted.is_hermitian()


@pytest.mark.parametrize("span", [(2, 2), (3, 1), (30, 21)])
@pytest.mark.parametrize("flux", [0, 7])
def test_lattices(gpu, span, flux):
    """All are but one: around a single cell under a gauge a hopping ends on its own site, which
    then has a complex energy."""
    X = tb.PartialLattice(tb.Honeycomb().add_hopping("A", 1, -2.7).add_hopping("A", 2, 0.13), span)
    if flux:
        K = np.zeros((3, 3))
        K[1, 0] = 2 * np.pi / flux
        X.set_gauge_linear(K)
    H = X.get_Hamiltonian_periodic_extend_bare_sparse([0 if flux else 1, 1], complex)
    cp, ri, v = H.to_csc()
    D = np.zeros(H.shape, dtype=complex)
    D[ri, np.repeat(np.arange(H.shape[0]), np.diff(cp))] = v
    expect = bool(np.max(np.abs(D - D.conj().T)) <= 1e-14)
    assert expect == (not (flux and span == (3, 1)))
    assert H.is_hermitian() == expect and tb.GreenFunction(2, H, -9.0, 9.5).scaled_HE.is_hermitian() == expect
