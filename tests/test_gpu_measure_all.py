"""qc_measure_all in one launch: the outcomes and the state that measuring the
qubits one after the other gives, for states below a warp's work, of a block's,
the largest that is measured so and one qubit more (which is measured qubit by
qubit), in both precisions.

The scales of the two ways are rounded from sums that may differ in their last
bit, so amplitudes agree to one unit of the precision a qubit."""
import ctypes as C

import numpy as np
import pytest

from qcs_gb300 import capi
from qcs_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def random_gates(A, c, n, seed):
    rng = W.Rng(seed)
    for _ in range(12 * n):
        t = rng.below(n)
        other = (t + 1 + rng.below(n - 1)) % n if n > 1 else t
        k = rng.below(5 if n > 1 else 3)
        if k == 0:
            A.qc_h(c, t)
        elif k == 1:
            A.qc_rx(c, t, rng.angle())
        elif k == 2:
            A.qc_rz(c, t, rng.angle())
        elif k == 3:
            A.qc_cnot(c, other, t)
        else:
            A.qc_cphase(c, other, t, rng.angle())


@pytest.mark.parametrize("prec,n", [(capi.C64, n) for n in (2, 5, 6, 7, 11, 12, 14, 15)] +
                         [(capi.C128, n) for n in (1, 4, 10, 13, 14)])
@pytest.mark.parametrize("kind", ["random", "basis"])
def test_measure_all_is_measuring_in_turn(prec, n, kind):
    A, libc = capi.api(), capi.libc()
    for seed in (1, 2, 3):
        got = []
        for together in (True, False):
            c = A.qc_create_ex(n, prec, capi.PHYSICAL, 0)
            A.qc_set_basis(c, (1 << n) - 2)
            if kind == "random":
                random_gates(A, c, n, 5 + n)
            libc.srand(seed)
            res = (C.c_int * n)()
            if together:
                A.qc_measure_all(c, res)
            else:
                for q in range(n):
                    res[q] = A.qc_measure(c, q)
            bits = list(res)
            index = sum(b << q for q, b in enumerate(bits))
            got.append((bits, A.qc_get_probability64(c, index),
                        A.qc_find_most_likely_state(c), libc.rand()))
            A.qc_destroy(c)
        assert got[0][0] == got[1][0]
        assert got[0][2:] == got[1][2:]
        eps = np.finfo(np.float32 if prec == capi.C64 else np.float64).eps
        assert abs(got[0][1] - got[1][1]) <= 2 * n * eps
        assert abs(got[0][1] - 1.0) <= 16 * n * eps
