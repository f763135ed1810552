"""Sums over moments split over 16 lanes: orders around one and two lane strides, points
around whole warps and CTAs, on and off the real axis, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,points", [(1, 1), (2, 3), (15, 2), (16, 8), (17, 9), (33, 7), (511, 130), (1024, 33)])
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
        assert np.all(np.abs(out - orc.green_imag_eval(g, mu, z)) <= tol)
