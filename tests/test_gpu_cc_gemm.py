"""The CUDA-core mu_nm GEMM at the edges of its tiles (64 x 32 outputs, 16 k a tile, 32 k a
sum, splits of 1,024 k and more) against FP64 products of the complex64 blocks."""
from __future__ import annotations

import numpy as np
import pytest

import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu
# of sum |L||R| per real part: 64 FP32 products and additions of a 32-term sum, 2^-24 each,
# and the float-float sum's 2^-40
BOUND = 64 * 2.0 ** -24 + 2.0 ** -40


@pytest.mark.parametrize("M,K", [(1, 1), (31, 15), (32, 16), (33, 17), (63, 32), (64, 33), (65, 48), (70, 1023),
                                 (97, 1025), (129, 3000), (5, 70000)])
def test_edges(gpu, M, K):
    rng = np.random.default_rng(M + K)
    L, R = ((rng.normal(size=(M, K)) + 1j * rng.normal(size=(M, K))).astype(np.complex64).astype(complex)
            for _ in range(2))
    mu = tb.mu_from_blocks(L, R, tensor=False)
    err = np.abs(mu - L.conj() @ R.T)
    assert np.all(err <= np.sqrt(2) * np.sqrt(2) * BOUND * (np.abs(L) @ np.abs(R).T))


@pytest.mark.parametrize("value", [np.inf, 1e39, 1e25, np.nan])
def test_infinities(gpu, value):
    """Infinities, values and products past FP32's range: infinite as their IEEE sums are, the
    rest of the matrix as without them."""
    rng = np.random.default_rng(3)
    L, R = ((np.abs(rng.normal(size=(3, 100))) + 0j) for _ in range(2))
    ref = L @ R.T
    L[1, 37] = value
    R[1, 37] = 1e25
    mu = tb.mu_from_blocks(L, R, tensor=False)
    assert np.isnan(mu[1, 1].real) if np.isnan(value) else np.isposinf(mu[1, 1].real)
    keep = np.ix_([0, 2], [0, 2])
    assert np.all(np.abs(mu[keep] - ref[keep]) <= 2 * (BOUND + 2.0 ** -23) * ref[keep].real)
