"""Kernels that start before the end of the kernel before them see all of its
results: gates one by one, runs of gates, read-outs and resets in a row without
a wait between them, at the sizes around which sweeps and tile passes start
early or not, against one run at a time with a wait after each call.  The same
kernels in the same order: equal bit for bit."""
import numpy as np
import pytest

from qcs_gb300 import capi
from qcs_gb300 import workloads as W
from tests.test_gpu_tiles import every_kind

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,sem,n", [(capi.C64, capi.PHYSICAL, n) for n in (5, 16, 17, 18, 19, 20)] +
                         [(capi.C128, capi.PHYSICAL, n) for n in (6, 15, 16, 18)] +
                         [(capi.C128, capi.REFERENCE, 15), (capi.C64, capi.REFERENCE, 18)])
def test_launches_in_a_row_wait_for_one_another(prec, sem, n):
    g = every_kind(n, 70 + n, 60)
    ops = list(zip(g.kinds, g.targets, g.controls, g.angles))
    got = []
    for wait in (False, True):
        with capi.State(n, prec, sem) as s:
            z = []
            for repeat in range(3):
                s.set_basis(repeat)
                for i, (k, t, c, a) in enumerate(ops):
                    s.apply_gate(k, t, c, a)
                    if wait:
                        s.synchronize()
                    if i % 20 == 19:
                        z.append(s.expect_z(i % n))
                s.phase_flip(3)
                if wait:
                    s.synchronize()
                for _ in range(3):
                    s.run(g)
                    if wait:
                        s.synchronize()
                z.append(s.norm_sq())
            got.append((np.array(z), s.amplitudes()))
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1], got[1][1])
    assert abs(got[0][0][-1] - 1.0) < 1e-3 or sem == capi.REFERENCE
