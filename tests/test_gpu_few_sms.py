"""Small solves under a limit on the SMs (a green context of 16): the cooperative launch of the
whole recursion is refused there, and the plan runs step by step with the same bits."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import tight_binding_gb300 as tb
from tight_binding_gb300 import capi

pytestmark = pytest.mark.gpu
SM_RESOURCE, DEFAULT_STREAM, NON_BLOCKING = 1, 1, 1        # CUDA's enumerators


@pytest.fixture
def sixteen_sms(gpu):
    """(stream, context) of 16 SMs through the driver's C interface."""
    cu = C.CDLL("libcuda.so.1")
    dev, count, desc, green, stream, ctx, old = C.c_int(), C.c_uint(1), *(C.c_void_p() for _ in range(5))
    whole, part, rest = (C.create_string_buffer(256) for _ in range(3))

    def call(name, *args):
        assert getattr(cu, name)(*args) == 0, name

    tb.device_count()
    tb.kernel_seq(8, tb.Jackson())                         # the primary context is current
    call("cuDeviceGet", C.byref(dev), 0)
    call("cuCtxGetCurrent", C.byref(old))
    call("cuDeviceGetDevResource", dev, whole, SM_RESOURCE)
    call("cuDevSmResourceSplitByCount", part, C.byref(count), whole, rest, 0, 16)
    call("cuDevResourceGenerateDesc", C.byref(desc), part, 1)
    call("cuGreenCtxCreate", C.byref(green), desc, dev, DEFAULT_STREAM)
    call("cuGreenCtxStreamCreate", C.byref(stream), green, NON_BLOCKING, 0)
    call("cuCtxFromGreenCtx", C.byref(ctx), green)
    capi.check(capi.lib().tbk_set_wait_limit(1 << 18))     # should a launch be let through after all
    yield stream, lambda on: call("cuCtxSetCurrent", ctx if on else old)
    capi.check(capi.lib().tbk_set_wait_limit(-1))
    call("cuCtxSetCurrent", old)
    call("cuStreamDestroy_v2", stream)
    call("cuGreenCtxDestroy", green)


@pytest.mark.parametrize("precision", ["fp64", "dd", "mixed"])
@pytest.mark.parametrize("doubling", [True, False])
def test_runs_in_steps(sixteen_sms, precision, doubling):
    stream, limit = sixteen_sms
    X = tb.PartialLattice(tb.Square().add_hopping("A", 1, 0.24), (128, 100))
    A = X.get_Hamiltonian_periodic_extend_bare_sparse([1, 1], float)
    kets = tb.bases_of_uniform_ampl_with_random_phases(A.shape[0], 8, 1)
    bras = kets if doubling else tb.bases_of_uniform_ampl_with_random_phases(A.shape[0], 8, 2)
    S = tb.KpmSolver(A, 8, precision, doubling)
    ref = S.run(40, bras, kets)
    for _ in range(3):                                     # steps, captured as a graph, replayed
        assert np.array_equal(S.run(40, bras, kets, stream), ref)
    limit(True)
    try:
        mu = tb.KpmSolver(A, 8, precision, doubling).run(40, bras, kets)
    finally:
        limit(False)
    assert np.array_equal(mu, ref)
    assert np.array_equal(S.run(40, bras, kets), ref)      # whole GPU: one launch again
