"""The batched kernel at the edges of its tiles and windows: instances smaller
than a thread's registers, exactly one tile, one qubit more (the smallest that
run in stages), more gates than the window of gates in shared memory holds
(256) and than one group may have, every gate kind, and every CTA size (which
also changes the registers a thread holds).

<Z_0> against the FP64 oracle to 1e-5, the bar of the other batch tests; the
results of one schedule equal another's bit for bit at the same tile size."""
import numpy as np
import pytest

from oracle import oracle as O
from qcs_gb300 import capi
from qcs_gb300 import workloads as W
from tests.test_gpu_tiles import every_kind

pytestmark = pytest.mark.gpu


def many_kinds(n, seed, count):
    if n > 1:
        return every_kind(n, seed, count, p_move=0.4)
    g = W.GateList()
    rng = W.Rng(seed)
    for _ in range(count):
        k = W.ONE_QUBIT_SET[rng.below(len(W.ONE_QUBIT_SET))]
        g.add(k, 0, -1, rng.angle() if k in W.PARAMETRIC else 0.0)
    return g


def test_batch_tile_edges_every_schedule():
    inst = [(n, many_kinds(n, n, 40 + 7 * n)) for n in (1, 2, 3, 4, 5, 6, 10, 11, 12, 13, 14)]
    # many gates on two qubits (one long group), and a long mixed list
    long_group = W.GateList()
    for i in range(700):
        long_group.add(W.CNOT if i % 2 else W.RX, 1, 0 if i % 2 else -1, 0.1 + 0.01 * i)
    inst += [(11, long_group), (12, many_kinds(12, 99, 900)), (4, W.GateList()), (15, W.GateList())]
    want = []
    for n, g in inst:
        with O.OracleState(n) as o:
            o.run(g)
            want.append(o.expect_z(0))
    seen = {}
    with capi.Batch(inst, shots=300, seed=9) as b:
        for schedule in ((256, 10, 2, 0), (512, 10, 1, 1), (1024, 10, 1, 0), (256, 12, 4, 0),
                         (512, 12, 2, 0), (1024, 13, 1, 0), (256, 13, 2, 0), (512, 14, 1, 0)):
            b.config(*schedule)
            z, samples, _ = b.run()
            np.testing.assert_allclose(z, want, atol=1e-5)
            for (n, _), s in zip(inst, samples):
                assert s.min() >= 0 and s.max() < 1 << n
            first = seen.setdefault(schedule[1], (z, samples))
            assert np.array_equal(samples, first[1]), schedule
            np.testing.assert_allclose(z, first[0], rtol=0, atol=1e-13)


@pytest.mark.parametrize("count", [1, 3, 40])
def test_batch_tickets_any_sharing_same_bits(count):
    # stages of 2 to 512 tiles (64 tickets at most) taken by one CTA, by queued
    # groups and by every CTA that comes free; more instances than one, and
    # fewer than CTAs
    inst = W.variational_batch(count, seed=7 + count, n_range=(11, 19), depth_range=(1, 5))
    inst[0] = (14, inst[0][1] if inst[0][0] <= 14 else many_kinds(14, 3, 60))
    with capi.Batch(inst, shots=200, seed=2) as b:
        for schedule, splits in (((256, 10, 2, 0), (27, 18, 10)), ((256, 13, 2, 1), (27, 15, 13))):
            for split in splits:
                b.config(*schedule)
                b.split(split)
                for repeat in range(2):
                    z, samples, _ = b.run()
                    key = (z.tobytes(), samples.tobytes())
                    if split == splits[0] and repeat == 0:
                        first = key
                    assert key == first, (schedule, split)
            for i in range(min(count, 3)):
                n, g = inst[i]
                with O.OracleState(n) as o:
                    o.run(g)
                    assert abs(o.expect_z(0) - z[i]) < 1e-5


def test_batch_readout_of_every_size_and_value():
    # blocks of 32, 64, ... amplitudes, one sampling tile to many; amplitudes
    # that are zero, below the smallest normal float, and all on one index
    small = W.GateList()
    for _ in range(3):
        small.add(W.RX, 3, -1, 2e-14)  # |a|^2 of the odd branches: 1e-28, 1e-56, ...
    small.add(W.RX, 0, -1, 1e-19)
    small.add(W.RX, 7, -1, 1e-22)
    inst = []
    for n in (1, 3, 5, 8, 13, 14, 15, 17, 19, 20):
        ones, spread = W.GateList(), W.GateList()
        for q in range(n):
            ones.add(W.X, q)
            spread.add(W.H, q)
        spread.add(W.RY, n - 1, -1, 0.7)
        inst += [(n, ones), (n, spread)]
    inst += [(9, small), (14, small), (16, small)]
    shots = 2000
    with capi.Batch(inst, shots=shots, seed=21) as b:
        z, samples, _ = b.run()
    for i, (n, g) in enumerate(inst):
        with O.OracleState(n) as o:
            o.run(g)
            assert abs(o.expect_z(0) - z[i]) < 1e-5, i
        s = samples[i]
        assert s.min() >= 0 and s.max() < 1 << n
        if g is small:
            assert not s.any()
        elif i % 2 == 0:
            assert (s == (1 << n) - 1).all()
        else:  # each low bit is fair: 6 standard deviations
            for q in range(n - 1):
                assert abs((s >> q & 1).mean() - 0.5) < 6 * 0.5 / np.sqrt(shots), (n, q)
