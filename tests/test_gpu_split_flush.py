"""The tensor-core mu_nm GEMM over K ranges of several register sums a CTA: 128 k an FP32 chunk,
32 chunks (4,096 k) a register sum, added into FP64 partial tiles, which every sum but a
CTA's first reads back."""
from __future__ import annotations

import numpy as np
import pytest

import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu
# of sum |L||R|: dropped lo lo products and lo rounding 2 x 2^-22; 48 FP32 accumulations of a
# chunk and 32 of a register sum, 2^-23 each; the complex64 rounding of the inputs 2 x 2^-24
BOUND = np.sqrt(2) * (2.0 ** -21 + 80 * 2.0 ** -23 + 2.0 ** -23)


# one row of output tiles, 2 CTAs wide: 152 SMs take K in 76 parts
@pytest.mark.parametrize("chunks,short", [(31, 0), (32, 0), (32, 1), (33, 0), (33, 127), (64, 0), (65, 45), (97, 31), (216, 0)])
@pytest.mark.parametrize("M", [2, 130])
@pytest.mark.parametrize("kind", ["independent", "equal", "drift"])
def test_flushes(gpu, M, chunks, short, kind):
    if M == 130:                                           # 2 x 2 tiles: half as many parts
        chunks = min(chunks, 65)
    K = (76 if M <= 128 else 38) * 128 * chunks - short
    rng = np.random.default_rng(chunks)
    L = (rng.standard_normal((M, K), np.float32) + 1j * rng.standard_normal((M, K), np.float32)).astype(np.complex128)
    if kind == "drift":                                    # from e^-6 to e^6 along k
        L *= np.exp(np.linspace(-6, 6, K))
    R = L[::-1] * (1 + 0.5j) if kind == "independent" else L
    mu = tb.mu_from_blocks(L, R, tensor=True)
    assert np.all(np.abs(mu - L.conj() @ R.T) <= BOUND * (np.abs(L) @ np.abs(R).T))
