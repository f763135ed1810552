"""The spectra from a moment matrix as one trigonometric series, against the oracle's double sums."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu


# sizes around the 16-row chunks, the 32-term lane stride of the series and the 4 energies of a CTA
@pytest.mark.parametrize("M,n_eps", [(1, 1), (2, 3), (15, 4), (16, 5), (17, 4), (33, 129), (65, 7), (300, 64)])
def test_series_equals_double_sum(gpu, M, n_eps):
    rng = np.random.default_rng(M)
    mu = rng.standard_normal((M, M)) + 1j * rng.standard_normal((M, M))
    eps = np.cos((np.arange(n_eps) + 0.5) * np.pi / n_eps) if n_eps > 1 else np.array([0.3])
    a = np.where(np.arange(M) == 0, 1.0, 2.0)
    w = np.outer(a, a) * np.abs(mu)
    s2 = 1 - eps ** 2
    idx = np.add.outer(np.arange(M), np.arange(M))
    # rounding of sums of at most 2M terms and of the angles q theta (q < 2M), on the absolute sums
    unit = 8 * (2 * M + 8) * np.finfo(float).eps
    tol_z = unit * (2 * w.sum() + np.sqrt(s2) * (w * idx).sum()) / s2 ** 2 / 2.5
    tol_s = unit * w.sum() / s2 / 3.0
    assert np.all(np.abs(tb.bastin_zeta(mu, eps, 2.5) - orc.bastin_zeta(mu, eps, 2.5)) <= tol_z)
    assert np.all(np.abs(tb.greenwood_sigma(mu, eps, 3.0) - orc.greenwood_sigma(mu, eps, 3.0)) <= tol_s)
