"""Batch read-outs of instances that live in shared memory, at the sizes where the
blocks that they are summed by change (8, 16 and 32 amplitudes, one block and many,
one sampling tile and several), with no shots and with many, alone and beside an
instance in a slot.

Hadamards on every qubit give each index the mass 2^-n, so a draw r of the documented
generator reads floor(r 2^n).  Each gate rounds an amplitude by at most 2^-24 and its
constant by 2^-25, a mass by twice that, so the running sums are within n 2^-22 of
exact ones: draws closer than that to an index's edge are left out.  <Z_0> is 0 (-1
with an X in place of the Hadamard on qubit 0) to the same bound."""
import numpy as np
import pytest

from qcs_gb300 import capi
from qcs_gb300 import workloads as W

pytestmark = pytest.mark.gpu

MASK = (1 << 64) - 1


def draw(seed, inst, shot):
    x = seed ^ (inst * 0xD1B54A32D192ED03 & MASK) ^ (shot * 0x8CB92BA72F3D8DD7 & MASK)
    x = (x + 0x9E3779B97F4A7C15) & MASK
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & MASK
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & MASK
    x ^= x >> 31
    return (x >> 11) * 2.0 ** -53


def instance(n, first):
    g = W.GateList()
    for q in range(n):
        g.add(first if q == 0 else W.H, q)
    return n, g


SIZES = [1, 2, 3, 4, 5, 8, 10, 11, 12, 13, 14]


@pytest.mark.parametrize("schedule", [(256, 14, 1, 0), (512, 14, 1, 0), (1024, 14, 1, 0),
                                      (256, 12, 2, 0), (256, 13, 2, 1)])
@pytest.mark.parametrize("extra", [0, 1])
def test_shots_and_z_of_small_instances(schedule, extra):
    sizes = SIZES + [16] * extra
    shots, seed = 300, 77
    with capi.Batch([instance(n, W.H) for n in sizes], shots=shots, seed=seed) as b:
        b.config(*schedule)
        z, samples, _ = b.run()
    assert np.max(np.abs(z)) <= 16 * 2.0 ** -22
    for i, n in enumerate(sizes):
        at = np.array([draw(seed, i, s) for s in range(shots)]) * 2.0 ** n
        clear = np.abs(at - np.rint(at)) > n * 2.0 ** (n - 22)
        assert clear.sum() > shots // 3
        assert np.array_equal(samples[i][clear], np.floor(at[clear]).astype(np.int64)), n


@pytest.mark.parametrize("schedule", [(256, 13, 2, 0), (512, 14, 1, 0), (1024, 12, 1, 0)])
def test_no_shots(schedule):
    sizes = SIZES + [15]
    first = [W.X if i % 2 else W.H for i in range(len(sizes))]
    with capi.Batch([instance(n, f) for n, f in zip(sizes, first)], shots=0, seed=1) as b:
        b.config(*schedule)
        z = b.run(want_samples=False)[0]
    want = np.array([-1.0 if f == W.X else 0.0 for f in first])
    assert np.max(np.abs(z - want)) <= 16 * 2.0 ** -22
