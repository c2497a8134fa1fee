"""Tile passes on finite states whose amplitudes overflow on the way: infinities
and the NaNs that follow from them lie where the gates one by one put them, in
tiles that come to overflow and, beside them, tiles that do not.

Tolerance: none (see test_gpu_tiles.py)."""
import numpy as np
import pytest

from qcs_gb300 import capi
from qcs_gb300 import workloads as W
from tests.test_gpu_tiles import FORMS, compare, every_kind, start

pytestmark = pytest.mark.gpu


def near_the_top(n, prec, seed, first, count):
    """A random state; `count` amplitudes from `first` on are near the largest number."""
    a = start(n, seed)
    top = float(np.finfo(np.float32 if prec == capi.C64 else np.float64).max)
    r = np.random.default_rng(seed)
    a[first:first + count] = top * (r.uniform(0.7, 0.99, count) + 1j * r.uniform(-0.99, 0.99, count))
    return a


@pytest.mark.parametrize("prec,sem", FORMS)
@pytest.mark.parametrize("n", [4, 9, 13, 17, 20])
def test_overflow_on_the_way(n, prec, sem):
    size = 1 << n
    for seed, first, count, gates in ((1, 0, 2, 6), (2, size - 3, 3, 40), (3, size // 2, 4, 150)):
        compare(n, prec, sem, every_kind(n, 40 * n + seed, gates),
                near_the_top(n, prec, seed, first, count))


@pytest.mark.parametrize("prec,sem", FORMS)
def test_overflow_by_each_kind_of_gate(prec, sem):
    """H makes an infinity; then each kind of gate, on the qubit and beside it."""
    n = 12
    for kind in (W.H, W.X, W.Y, W.Z, W.P, W.RX, W.RY, W.RZ, W.CNOT, W.CPHASE, W.I):
        g = W.GateList()
        g.add(W.H, 1)
        for t in (1, 0, n - 1):
            c = (t + 1) % n if kind in (W.CNOT, W.CPHASE) else -1
            g.add(kind, t, c, 0.7 if kind in W.PARAMETRIC else 0.0)
            g.add(kind, t, c, 0.0)  # an angle of 0: what the sweeps leave out
        g.add(W.RY, 3, -1, 0.2)
        compare(n, prec, sem, g, near_the_top(n, prec, 5, 0, 6))


@pytest.mark.parametrize("prec,sem", FORMS)
@pytest.mark.parametrize("n", [5, 13, 20])
def test_passes_of_moves_alone(n, prec, sem):
    """X and CNOT take no arithmetic; the products with zeros of their sweeps make
    NaNs of an infinity all the same."""
    compare(n, prec, sem, every_kind(n, 900 + n, 12, 1.0), start(n, 7))
    compare(n, prec, sem, every_kind(n, 900 + n, 12, 1.0), start(n, 8, bad=True))
