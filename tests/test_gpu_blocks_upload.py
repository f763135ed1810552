"""mu_from_blocks takes its blocks up several at a time (32 MB): values at the edges of such a
group, and the time of many small blocks."""
from __future__ import annotations

import time

import numpy as np
import pytest

import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu
# of sum |L||R|, as in test_gpu_split_gemm.py with 32 additions of a register sum; the CUDA-core
# form makes 32 of a chunk
BOUND = np.sqrt(2) * (2.0 ** -21 + 80 * 2.0 ** -23 + 2.0 ** -23)


# groups of 34 blocks, of 2, of 1; all blocks in one group
@pytest.mark.parametrize("M,K", [(34, 61_000), (35, 61_000), (69, 61_000), (5, 1_000_000), (3, 2_100_000), (200, 9)])
@pytest.mark.parametrize("tensor", [True, False])
def test_groups(gpu, M, K, tensor):
    rng = np.random.default_rng(M)
    L, R = ((rng.standard_normal((M, K), np.float32) + 1j * rng.standard_normal((M, K), np.float32)).astype(complex)
            for _ in range(2))
    L *= 10.0 ** rng.integers(-9, 9, size=(M, 1))
    mu = tb.mu_from_blocks(L, R, tensor=tensor)
    assert np.all(np.abs(mu - L.conj() @ R.T) <= BOUND * (np.abs(L) @ np.abs(R).T))


def test_not_finite_in_a_later_group(gpu):
    rng = np.random.default_rng(0)
    L, R = (rng.normal(size=(40, 61_000)) + 0j for _ in range(2))
    R[38, 60_999] = np.nan
    assert np.array_equal(tb.mu_from_blocks(L, R, tensor=True), tb.mu_from_blocks(L, R, tensor=False), equal_nan=True)


@pytest.mark.parametrize("tensor", [True, False])
def test_many_small_blocks(gpu, tensor):
    def best(M):
        L = np.ones((M, 7), dtype=complex)
        t = []
        for _ in range(5):
            t0 = time.perf_counter()
            tb.mu_from_blocks(L, L, tensor=tensor)
            t.append(time.perf_counter() - t0)
        return min(t)

    best(1)
    assert best(400) <= 15 * best(1)                       # one by one: 50 to 130 times
