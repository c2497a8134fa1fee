"""qc_measure_all under REFERENCE semantics: outcomes, state and second buffer (which
a phase flip brings back) as by measuring the qubits in turn.

Amplitudes agree to one unit of the precision a qubit: the scales of the two ways are
rounded from sums that may differ in their last bit."""
import ctypes as C

import numpy as np
import pytest

from qcs_gb300 import capi
from tests.test_gpu_measure_all import random_gates

pytestmark = pytest.mark.gpu


def amplitudes(A, c, n):
    out = np.zeros(2 << n)
    rc = capi.lib().qcs_cuda_read_amplitudes(A.qc_cuda_state(c), 0, 1 << n,
                                             out.ctypes.data_as(C.POINTER(C.c_double)))
    assert rc == capi.OK
    return out


@pytest.mark.parametrize("prec,n", [(capi.C64, 2), (capi.C64, 7), (capi.C64, 14), (capi.C128, 5),
                                    (capi.C128, 13), (capi.C128, 14)])
def test_measure_all_is_measuring_in_turn(prec, n):
    A, libc = capi.api(), capi.libc()
    eps = np.finfo(np.float32 if prec == capi.C64 else np.float64).eps
    for seed in (1, 2):
        got = []
        for together in (True, False):
            c = A.qc_create_ex(n, prec, capi.REFERENCE, 0)
            A.qc_set_basis(c, 1)
            random_gates(A, c, n, 9 + n)
            libc.srand(seed)
            res = (C.c_int * n)()
            if together:
                A.qc_measure_all(c, res)
            else:
                for q in range(n):
                    res[q] = A.qc_measure(c, q)
            state = amplitudes(A, c, n)
            assert capi.lib().qcs_cuda_phase_flip(A.qc_cuda_state(c), 0) == capi.OK
            got.append((list(res), state, amplitudes(A, c, n), libc.rand()))
            A.qc_destroy(c)
        assert got[0][0] == got[1][0] and got[0][3] == got[1][3]
        # the reference's gates do not keep the norm: relative to the largest amplitude
        top = np.max(np.abs(got[1][1]))
        assert np.max(np.abs(got[0][1] - got[1][1])) <= 2 * n * eps * top
        # the second buffer is untouched by both but for the flipped amplitude
        assert np.array_equal(got[0][2][2:], got[1][2][2:])
        assert np.max(np.abs(got[0][2][:2] - got[1][2][:2])) <= 2 * n * eps * top
