"""Spectral ranges of matrices with few distinct eigenvalues: the recursion ends with them."""
from __future__ import annotations

import time

import numpy as np
import pytest

import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu


def _clusters(n, k):
    """n / k separate rings of k sites, hopping 1: at most k // 2 + 1 distinct eigenvalues."""
    j = np.arange(n)
    a, b = j // k * k + (j + 1) % k, j // k * k + (j - 1) % k
    ri = np.stack([np.minimum(a, b), np.maximum(a, b)], axis=1).ravel().astype(np.int32)
    return tb.SparseMatrix.from_csc(n, n, (2 * np.arange(n + 1)).astype(np.int32), ri, np.ones(2 * n))


@pytest.mark.parametrize("k,iters", [(k, i) for k in (4, 8, 40, 130) for i in (4, 5, 16, 17, 64, 65, 200, 400)
                                     if i > k // 2 + 1])
def test_range(gpu, k, iters):
    e0, e1, r0, r1 = tb.spectral_range(_clusters(520, k), iters=iters, seed=1)
    assert abs(e0 + 2) <= 1e-10 and abs(e1 - 2) <= 1e-10 and max(r0, r1) <= 1e-10


def test_does_not_run_all_iterations(gpu):
    H = _clusters(200_000, 4)

    def ms(iters):
        best = np.inf
        for _ in range(3):
            t = time.perf_counter()
            tb.spectral_range(H, iters=iters)
            best = min(best, 1e3 * (time.perf_counter() - t))
        return best

    ms(4)
    assert ms(20_000) <= 4 * ms(16) + 4.0                  # 20,000 iterations take some 200 ms
