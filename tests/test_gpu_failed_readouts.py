"""A read-out that follows one that failed returns its own value.

A launch can be reported as failed although the kernel runs (an older error of
the thread; the injected failure here, which is reported after the launch).  Its
call returns at once, so the next read-out starts while that kernel is still at
work.  On 28 qubits a read-out runs for longer than the host takes to start the
next one.

Tolerance: none.  The value is that of the same call without a failure before it,
and every read-out gives the same bits each time."""
import ctypes as C

import pytest

from qcs_gb300 import capi
from qcs_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def fail(call):
    """`call` with its first launch reported as failed."""
    L = capi.lib()
    L.qcs_cuda_debug_inject(2, 1)
    try:
        with pytest.raises(capi.QcsCudaError) as e:
            call()
        assert e.value.status == capi.ELAUNCH
    finally:
        L.qcs_cuda_debug_inject(0, 0)


@pytest.mark.parametrize("prec,n", [(capi.C64, 28), (capi.C128, 24)])
def test_the_next_readout_returns_its_own_value(prec, n):
    with capi.State(n, prec) as s:
        for q in range(n):
            s.apply_gate(W.RY, q, -1, 0.3 + 0.05 * q)
        calls = {"norm": s.norm_sq, "p0": lambda: s.prob_zero(3), "z": lambda: s.expect_z(n - 1),
                 "argmax": s.argmax, "probability": lambda: s.probability(5)}
        value = {name: call() for name, call in calls.items()}
        for before, failing in calls.items():
            for after, call in calls.items():
                fail(failing)
                assert call() == value[after], (before, after)


@pytest.mark.parametrize("prec,n", [(capi.C64, 2), (capi.C64, 10), (capi.C64, 14),
                                    (capi.C128, 13)])
def test_measure_all_after_a_failure_leaves_the_state_to_the_other_qubits(prec, n):
    """The failing launch reads 0 for qubit 0 and does not collapse the state; the
    other qubits are measured one by one."""
    A, L = capi.api(), capi.lib()
    c = A.qc_create_ex(n, prec, capi.PHYSICAL, 0)
    A.qc_set_basis(c, (1 << n) - 1)
    bits = (C.c_int * n)()
    L.qcs_cuda_debug_inject(2, 1)
    A.qc_measure_all(c, bits)
    L.qcs_cuda_debug_inject(0, 0)
    assert list(bits) == [0] + [1] * (n - 1)
    assert A.qc_get_probability64(c, (1 << n) - 1) == 1.0
    A.qc_measure_all(c, bits)
    assert list(bits) == [1] * n
    A.qc_destroy(c)
