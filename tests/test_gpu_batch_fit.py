"""Batch schedules name CTAs that an SM holds: what the autotuner chooses is what
runs, and a schedule of more runs as one of fewer, with the same results."""
import ctypes as C

import numpy as np
import pytest

from qcs_gb300 import capi
from qcs_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(8))
def test_the_autotuner_chooses_what_runs(seed):
    with capi.Batch(W.variational_batch(8, seed, n_range=(6, 10)), shots=4) as b:
        chosen = (C.c_int * 4)()
        assert capi.lib().qcs_cuda_batch_autotune(b._h, 1, chosen) == capi.OK
        s = b.schedule()
        assert list(chosen)[:3] == [s["threads"], s["tile_q"], s["ctas_per_sm"]]


@pytest.mark.parametrize("threads,tile_q,more", [(256, 12, 4), (512, 12, 2), (256, 13, 2)])
def test_a_schedule_of_more_runs_as_one_that_fits(threads, tile_q, more):
    with capi.Batch(W.variational_batch(12, 3, n_range=(8, 15)), shots=64) as b:
        b.config(threads, tile_q, more, 0)
        fits = b.schedule()["ctas_per_sm"]
        z, samples, _ = b.run()
        assert 1 <= fits <= more
        b.config(threads, tile_q, fits, 0)
        assert b.schedule()["ctas_per_sm"] == fits
        z2, samples2, _ = b.run()
    assert np.array_equal(z, z2) and np.array_equal(samples, samples2)
