"""kubo_last_timing where a tensor-core GEMM is discarded (values past FP16's range) and the
result formed on the CUDA cores: each phase counts its own work."""
from __future__ import annotations

import numpy as np
import pytest

import tight_binding_gb300 as tb

pytestmark = pytest.mark.gpu


def _timings(call):
    out = []
    for tensor in (False, True):
        call(tensor)
        call(tensor)
        out.append(tb.kubo_last_timing())
    return out


def test_kubo_mu(gpu):
    X = tb.PartialLattice(tb.Square().add_hopping("A", 1, 1.0), (40, 40))
    H = X.get_Hamiltonian_periodic_extend_bare_sparse([1, 1], float)
    A = tb.GreenFunction(2, H, -3.5, 3.5).scaled_HE        # spectrum beyond [-1, 1]: the blocks grow
    v = tb.commutator(A, X.op_position(0))
    plain, tensor = _timings(lambda t: tb.kubo_mu(A, v, v, M=40, R=5, seed=3, tensor=t))
    assert tensor["gemm_flops"] == plain["gemm_flops"] and tensor["chunks"] == plain["chunks"]
    assert tensor["block_bytes"] > 1.8 * plain["block_bytes"]
    # 80 steps of 3 us or more build the blocks again
    assert tensor["ms_gemm"] <= 2 * plain["ms_gemm"] + 0.03
    assert tensor["ms_blocks"] >= 1.2 * plain["ms_blocks"]


def test_mu_from_blocks(gpu):
    rng = np.random.default_rng(0)
    L = rng.normal(size=(40, 60_000)) + 0j
    L[3, 5] = np.inf
    plain, tensor = _timings(lambda t: tb.mu_from_blocks(L, L, tensor=t))
    assert tensor["gemm_flops"] == plain["gemm_flops"]
    assert tensor["ms_gemm"] <= 2 * plain["ms_gemm"] + 0.03   # without the 77 MB uploaded again
