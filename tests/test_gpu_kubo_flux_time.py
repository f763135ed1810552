"""A Kubo solve under a flux whose rows repeat in too many classes: looking for them must not
cost more than the solve."""
from __future__ import annotations

import time

import numpy as np
import pytest

import tight_binding_gb300 as tb
from tight_binding_gb300.serving import model_bounds, model_cell

pytestmark = pytest.mark.gpu


def test_host_and_set_up_time(gpu):
    X = tb.PartialLattice(model_cell("kagome"), (261, 259))
    K = np.zeros((3, 3))
    K[1, 0] = 2 * np.pi / 16
    X.set_gauge_linear(K)
    H = X.get_Hamiltonian_periodic_extend_bare_sparse([0, 1], complex)
    A = tb.GreenFunction(2, H, *model_bounds("kagome", 1.0)).scaled_HE
    v = tb.commutator(A, X.op_position(0))
    rest = np.inf
    for _ in range(4):
        t = time.perf_counter()
        tb.kubo_mu(A, v, None, v, None, M=40, R=4, seed=3, tensor=True)
        T = tb.kubo_last_timing()
        rest = min(rest, 1e3 * (time.perf_counter() - t) - T["ms_blocks"] - T["ms_gemm"])
    assert rest <= 3.0                                     # 10 ms and more while the class table overflowed


@pytest.mark.parametrize("n", [1, 127, 128, 600, 5000])
def test_number_of_classes(gpu, n):
    """Rows of n different values: two classes each (the offset), up to 255; the ELL form beyond."""
    rows = 20_000
    j = np.arange(rows)
    v = 1.0 + (j // 2 % n) / 1024.0                        # pairs j, j ^ 1 with one value
    A = tb.SparseMatrix.from_csc(rows, rows, np.arange(rows + 1, dtype=np.int32), (j ^ 1).astype(np.int32), v)
    got = A.row_classes()
    expect = 2 * n if 2 * n <= 255 else 0                  # offsets +1 and -1
    assert got == expect
