"""Resolvent sums far outside [-1, 1], where the powers of z - i sqrt(1 - z^2) outgrow the
coefficients they belong to, against the oracle's recurrence."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 4, 12, 16, 17, 40, 512, 1024])
def test_matches_oracle(gpu, n):
    rng = np.random.default_rng(n)
    mu, g = rng.normal(size=n), orc.kernel_seq(orc.K_LORENTZ, n, 4.0)
    x = np.array([1.0001, 1.3, 2.0, 5.0, 40.0, 1e6, 1e12, 1e18, 1e19, 1e20, 1e21, 1e25, 1e30, 1e40])
    z = np.concatenate([x, -x, x * (1 + 0.3j), x * (-1 + 0.1j), x * 1j, x - 1j, -x * 1j]).astype(complex)
    zz = np.ascontiguousarray(np.stack([z.real, z.imag], 1))
    out = np.zeros(len(z))
    tb.capi.check(tb.capi.lib().tbk_green_imag_eval(n, g.ctypes.data, mu.ctypes.data, len(z), zz.ctypes.data,
                                                    out.ctypes.data, None))
    ref = orc.green_imag_eval(g, mu, z)
    with np.errstate(all="ignore"):
        s1 = np.sqrt(1 - z * z)
        w = np.abs(z - 1j * s1)
        size = np.array([np.sum(np.abs(g * mu) * 2 / abs(s) * np.exp(np.log(a) * np.arange(n))) for s, a in zip(s1, w)])
        # n products of 4 roundings, the root, and z - i s1 where it cancels (w is 1 / |2 z| there)
        tol = (8 * (n + 8) * np.finfo(float).eps) * size + 8 * np.finfo(float).eps * np.abs(z) * 2 / np.abs(s1) * n * np.abs(g * mu).sum() * (w < 1)
    fin = np.isfinite(ref) & np.isfinite(size)
    assert fin.sum() >= (len(z) // 4 if n <= 40 else 10)
    assert np.all(np.isfinite(out[fin])) and np.all(np.abs(out - ref)[fin] <= tol[fin])
