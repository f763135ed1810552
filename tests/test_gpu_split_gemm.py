"""The tensor-core mu_nm GEMM on FP16-pair stores: edges of its tiles (128 x 128 outputs,
32 k a tile, 128 k a chunk, 2,048 k a register sum), block scales, values out of range."""
from __future__ import annotations

import numpy as np
import pytest

import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu
# of sum |L||R|: dropped lo lo products and lo rounding 2 x 2^-22; 48 FP32 accumulations of a
# chunk and 16 of a register sum, 2^-23 each; the complex64 rounding of the inputs 2 x 2^-24
BOUND = 2.0 ** -21 + 64 * 2.0 ** -23 + 2.0 ** -23


@pytest.mark.parametrize("M,K", [(1, 1), (2, 31), (127, 32), (128, 33), (129, 127), (130, 128), (200, 129),
                                 (256, 2047), (257, 2048), (65, 2049), (300, 5000)])
def test_edges(gpu, M, K):
    rng = np.random.default_rng(M * 7919 + K)
    L, R = (rng.normal(size=(M, K)) + 1j * rng.normal(size=(M, K)) for _ in range(2))
    # blocks of very different size: every block has its own scale
    L *= 10.0 ** rng.integers(-12, 12, size=(M, 1))
    R *= 10.0 ** rng.integers(-12, 12, size=(M, 1))
    mu = tb.mu_from_blocks(L, R, tensor=True)
    err = np.abs(mu - L.conj() @ R.T)
    assert np.all(err <= BOUND * np.sqrt(2) * (np.abs(L) @ np.abs(R).T))


def test_zero_and_spike_blocks(gpu):
    M, K = 140, 700
    L = np.zeros((M, K), complex)
    R = np.zeros((M, K), complex)
    L[np.arange(M), np.arange(M) * 5] = 1e4 - 3j
    R[3:, :] = 1e-7j
    mu = tb.mu_from_blocks(L, R, tensor=True)
    assert np.all(np.abs(mu - L.conj() @ R.T) <= BOUND * np.sqrt(2) * (np.abs(L) @ np.abs(R).T))
    assert np.all(mu[:, :3] == 0)


@pytest.mark.parametrize("bad", [np.inf, np.nan, 1e30])
def test_values_out_of_range(gpu, bad):
    """A spike of 10^30 fits its block's own scale; infinities and NaN give what the
    complex64 path gives."""
    rng = np.random.default_rng(1)
    L, R = (rng.normal(size=(40, 300)) + 0j for _ in range(2))
    L[7, 11] = bad
    a, b = tb.mu_from_blocks(L, R, tensor=True), tb.mu_from_blocks(L, R, tensor=False)
    if np.isfinite(bad):
        assert np.all(np.abs(a - L.conj() @ R.T) <= BOUND * np.sqrt(2) * (np.abs(L) @ np.abs(R).T))
    else:
        assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("which", ["bastin", "greenwood"])
@pytest.mark.parametrize("recursion", ["mixed", "dd", "fp64"])
def test_diverging_recursion_falls_back(gpu, recursion, which):
    """Bounds inside the spectrum: the blocks grow past FP16's range, and the tensor path
    gives the bits of the complex64 stores and CUDA-core GEMM."""
    X = tb.PartialLattice(tb.Square().add_hopping("A", 1, 1.0), (12, 10))
    H = X.get_Hamiltonian_periodic_extend_bare_sparse([1, 1], float)
    A = tb.GreenFunction(2, H, -2.0, 2.0).scaled_HE          # spectrum [-2, 2] after the rescale
    v = tb.commutator(A, X.op_position(0))
    ops = (None, None, v, v) if which == "bastin" else (v, v, None, None)
    a = tb.kubo_mu(A, *ops, 24, 5, seed=3, tensor=True, recursion=recursion)
    b = tb.kubo_mu(A, *ops, 24, 5, seed=3, tensor=False, recursion=recursion)
    assert np.max(np.abs(b)) > 1e12 and np.array_equal(a, b)
