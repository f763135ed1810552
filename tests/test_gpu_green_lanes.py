"""Resolvent sums by 1, 4 and 16 lanes a point (chosen by the numbers of moments and points)
against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,points", [(1, 20_000), (2, 4_001), (3, 30_000), (4, 9_000), (5, 8_003), (63, 40_001), (64, 3_000),
                                      (130, 9_999), (512, 257), (511, 12_345), (512, 120_001), (17, 1_500)])
def test_matches_oracle(gpu, n, points):
    rng = np.random.default_rng(n)
    mu, g = rng.normal(size=n), orc.kernel_seq(orc.K_LORENTZ, n, 4.0)
    for im in (0.0, 0.02):
        z = np.linspace(-0.97, 0.95, points) + 1j * im
        zz = np.ascontiguousarray(np.stack([z.real, z.imag], 1))
        out = np.zeros(points)
        tb.capi.check(tb.capi.lib().tbk_green_imag_eval(n, g.ctypes.data, mu.ctypes.data, points, zz.ctypes.data,
                                                       out.ctypes.data, None))
        # n steps of a rotation, on the absolute sum of the terms (|alpha| <= 2 / |sqrt(1 - z^2)|)
        tol = 16 * (n + 8) * np.finfo(float).eps * 2 / np.abs(np.sqrt(1 - z * z)) * np.abs(g * mu).sum()
        some = np.unique(np.concatenate([rng.integers(0, points, 300), [0, points - 1]]))
        assert np.all(np.abs(out[some] - orc.green_imag_eval(g, mu, z[some])) <= tol[some])
    # a prefix of the points takes other lanes: the same sums
    k = 100
    few = np.zeros(k)
    tb.capi.check(tb.capi.lib().tbk_green_imag_eval(n, g.ctypes.data, mu.ctypes.data, k, zz.ctypes.data, few.ctypes.data,
                                                   None))
    assert np.all(np.abs(few - out[:k]) <= 2 * tol[:k])
