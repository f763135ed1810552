"""The scale of FP16-pair stores where an operator (nearly) vanishes on the start vectors but
not on T_m of them, against complex128 blocks and an FP64 product."""
from __future__ import annotations

import numpy as np
import pytest

import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu
# of |L_m||R_n|: dropped lo lo products and lo rounding 2 x 2^-22; 48 FP32 accumulations of a
# chunk and at most 32 of a register sum, 2^-23 each; the complex64 rounding of the stored values 2 x 2^-24
BOUND = np.sqrt(2) * (2.0 ** -21 + 80 * 2.0 ** -23 + 2.0 ** -23)


def _system(cell, span):
    X = tb.PartialLattice(cell.add_hopping("A", 1, 1.0), span)
    X.set_scalar_values(np.random.default_rng(2).random(X.get_total_number()) - 0.5)
    H = X.get_Hamiltonian_periodic_extend_bare_sparse([1, 1], float)
    return X, tb.GreenFunction(2, H, -5.0, 5.0).scaled_HE


def _kets(n, R, sites, amplitude):
    rng = np.random.default_rng(7)
    k = np.zeros((n, R), dtype=complex, order="F")
    k[sites] = amplitude * np.exp(2j * np.pi * rng.random((len(sites), R)))
    return k


def _check(A, V, kets, gain, M=40, **form):
    mu = tb.kubo_mu(A, V, None, V, None, M, kets=kets, tensor=True, **form)
    flops = tb.kubo_last_timing()["gemm_flops"]
    form.pop("fuse_ops", None), form.pop("both_sides", None)
    ref = tb.kubo_mu(A, V, None, V, None, M, kets=kets, fp64_blocks=True, **form)
    norm = np.sqrt(np.diag(ref).real)
    # a value's lo half ends at 2^-25 over the scale: 2^-31 of gain times the kets' rms
    floor = 2.0 ** -31 * gain * np.sqrt(2) * np.linalg.norm(kets)
    assert norm.max() > 0.01 * np.linalg.norm(kets)
    assert np.all(np.abs(mu - ref) <= BOUND * np.outer(norm, norm) + floor * np.add.outer(norm, norm) + floor ** 2)
    return flops


@pytest.mark.parametrize("recursion", ["mixed", "dd", "fp64"])
@pytest.mark.parametrize("amplitude", [1.0, 1e-4, 1e-8])
def test_projector_away_from_the_kets(gpu, amplitude, recursion):
    """Blocks of one checkerboard colour, kets on the other."""
    X, A = _system(tb.Square(), (24, 20))
    n = A.shape[0]
    (_, a, x), (_, b, y) = (X.op_position(k).to_csc() for k in range(2))
    at = np.zeros((n, 2))
    at[a, 0], at[b, 1] = x, y
    even = np.flatnonzero(np.rint(at.sum(axis=1)).astype(int) % 2 == 0)
    odd = np.setdiff1d(np.arange(n), even)
    cp = np.zeros(n + 1, dtype=np.int32)
    cp[even + 1] = 1
    V = tb.SparseMatrix.from_csc(n, n, np.cumsum(cp, dtype=np.int32), even.astype(np.int32), np.ones(len(even)))
    plain = _check(A, V, _kets(n, 5, even, amplitude), 1.0, recursion=recursion)
    assert _check(A, V, _kets(n, 5, odd, amplitude), 1.0, recursion=recursion) == plain
    # a first block of 1e-30 of the later ones stays on the tensor cores
    kets = _kets(n, 5, odd, amplitude)
    kets[even] = 1e-30 * amplitude
    assert _check(A, V, kets, 1.0, recursion=recursion) == plain


@pytest.mark.parametrize("form", [{}, {"fuse_ops": True}, {"fuse_ops": True, "both_sides": True}])
@pytest.mark.parametrize("recursion", ["mixed", "dd"])
def test_velocity_on_sites_without_x_bonds(gpu, recursion, form):
    """Lieb lattice, kets on the sites bonded only along y."""
    X, A = _system(tb.Lieb(), (14, 11))
    V = tb.commutator(A, X.op_position(0))
    n = A.shape[0]
    cp, ri, v = V.to_csc()
    rows = np.bincount(ri, np.abs(v), minlength=n)
    cols = np.bincount(np.repeat(np.arange(n), np.diff(cp)), np.abs(v), minlength=n)
    still = np.flatnonzero(cols == 0)
    assert len(still) == n // 3
    _check(A, V, _kets(n, 4, still, 1e-5), rows.max(), recursion=recursion, **form)
