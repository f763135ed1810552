"""The spectra at the outermost nodes, where the weights 1/(1 - e^2) and 1/(1 - e^2)^2 show how 1 - e^2
was rounded."""
from __future__ import annotations

import numpy as np
import pytest

import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [64, 1024, 4096])
def test_weights(gpu, N):
    eps = tb.chebyshev_nodes(N)
    mu = np.zeros((3, 3), dtype=complex)
    mu[0, 0] = 2.0                                         # Gamma_00 = 2 e: no sums, the weights alone
    q = 1.0 - eps * eps
    sigma, zeta = tb.greenwood_sigma(mu, eps, 3.0), tb.bastin_zeta(mu, eps, 3.0)
    s0, z0 = -1.0 / q, eps / (q * q)
    # up to constant factors, which the middle of the band gives; a dozen roundings
    m = N // 4
    assert np.max(np.abs(sigma / s0 / (sigma[m] / s0[m]) - 1)) <= 12 * 2.0 ** -52
    z = zeta.real
    assert np.max(np.abs(z / z0 / (z[m] / z0[m]) - 1)[np.abs(eps) > 0.01]) <= 12 * 2.0 ** -52
