"""Plain gate lists run in shared-memory tiles (tiles.cu): the same values,
bit for bit, as the gates applied one by one through the sweeps, at the edges
of the tiles (states smaller than one, exactly one, a few), where passes end
for want of room (gates, groups, flips), with controls and diagonal targets
outside the tile, and with infinities and NaNs in the state.

Tolerance: none.  Every product and sum is the sweeps', in their order; a
product with an exact 0 or 1 is left out, which changes at most the sign of a
zero, and zeros compare equal."""
import numpy as np
import pytest

from qcs_gb300 import capi
from qcs_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def every_kind(n, seed, count, p_move=0.25):
    """Random gates of every kind; p_move: the share of X and CNOT."""
    rng = W.Rng(seed)
    kinds = (W.H, W.Y, W.Z, W.P, W.RX, W.RY, W.RZ, W.CPHASE, W.I)
    g = W.GateList()
    for _ in range(count):
        t = rng.below(n)
        if rng.uniform() < p_move:
            k = W.X if rng.uniform() < 0.3 else W.CNOT
        else:
            k = kinds[rng.below(len(kinds))]
        c = -1
        if k in (W.CNOT, W.CPHASE):
            c = (t + 1 + rng.below(n - 1)) % n
        g.add(k, t, c, rng.angle() if k in W.PARAMETRIC else 0.0)
    return g


def start(n, seed, bad=False):
    r = np.random.default_rng(seed)
    a = r.normal(size=1 << n) + 1j * r.normal(size=1 << n)
    a /= np.linalg.norm(a)
    if bad:
        a[r.integers(0, 1 << n, 2)] = complex(np.inf, 0.5), complex(0.25, np.nan)
    return a


def one_by_one(s, g):
    for k, t, c, a, i in zip(g.kinds, g.targets, g.controls, g.angles, g.indices):
        if k == W.PHASE_FLIP:
            s.phase_flip(i)
        elif k == W.DIFFUSION:
            s.diffusion()
        else:
            s.apply_gate(k, t, c, a)


def compare(n, prec, sem, g, init):
    with capi.State(n, prec, sem) as a, capi.State(n, prec, sem) as b:
        a.set_amplitudes(init)
        b.set_amplitudes(init)
        one_by_one(a, g)
        b.run(g)
        x, y = a.amplitudes().view(np.float64), b.amplitudes().view(np.float64)
        assert np.array_equal(x, y, equal_nan=True)
        # the second buffer holds the state before the last gate
        if sem == capi.REFERENCE:
            a.phase_flip(1)
            b.phase_flip(1)
            x, y = a.amplitudes().view(np.float64), b.amplitudes().view(np.float64)
            assert np.array_equal(x, y, equal_nan=True)


FORMS = [(capi.C64, capi.PHYSICAL), (capi.C128, capi.PHYSICAL), (capi.C64, capi.REFERENCE),
         (capi.C128, capi.REFERENCE)]


@pytest.mark.parametrize("prec,sem", FORMS)
@pytest.mark.parametrize("n", [3, 4, 5, 9, 10, 11, 12, 13, 17])
def test_tiles_equal_sweeps(n, prec, sem):
    compare(n, prec, sem, every_kind(n, 100 + n, 300), start(n, n))


@pytest.mark.parametrize("prec,sem", FORMS)
def test_passes_that_end_full(prec, sem):
    """Many gates on few qubits (128 a pass), many moves (32 flips a pass)
    and targets that never repeat (groups)."""
    n = 13
    few = every_kind(4, 7, 300, 0.0)
    moves = every_kind(n, 8, 300, 1.0)
    wide = W.GateList()
    for rep in range(20):
        for q in range(n):
            wide.add((W.H, W.RX, W.RY, W.Y)[(rep + q) % 4], q, -1, 0.1 * rep + 0.3)
    for g in (few, moves, wide):
        compare(n, prec, sem, g, start(n, 3))


@pytest.mark.parametrize("prec,sem", FORMS)
def test_flips_and_diffusions_between_gates(prec, sem):
    n = 12
    g = W.GateList()
    for rep in range(3):
        g.extend(every_kind(n, 20 + rep, 30))
        g.add(W.PHASE_FLIP, index=77 + rep)
        g.add(W.X, rep)
        g.add(W.PHASE_FLIP, index=3)
    g.extend(W.qft_gates(n))
    compare(n, prec, sem, g, start(n, 4))


@pytest.mark.parametrize("prec,sem", FORMS)
@pytest.mark.parametrize("n", [6, 13])
def test_infinities_and_nans_spread_as_in_the_sweeps(n, prec, sem):
    compare(n, prec, sem, every_kind(n, 31, 12), start(n, 5, bad=True))
    compare(n, prec, sem, every_kind(n, 32, 60), start(n, 6, bad=True))


@pytest.mark.parametrize("sem", [capi.PHYSICAL, capi.REFERENCE])
@pytest.mark.parametrize("n", [4, 8, 9, 16, 17, 18])
def test_every_split_of_a_complex128_tile(n, sem):
    """4, 8 and 16 amplitudes a thread, tiles of 2^9 and 2^10; groups of few
    qubits (more groups than a pass takes), phases with conditions on every
    pair of register bits, and tiles with an infinity or a NaN."""
    wide = W.GateList()
    for rep in range(12):
        for q in range(n):
            wide.add(W.RY, q, -1, 0.3 + 0.1 * rep + 0.01 * q)
    for q in range(n):
        for p in range(n):
            if p != q:
                wide.add(W.CPHASE, q, p, 0.2 + 0.03 * q + 0.005 * p)
                wide.add(W.RX, p, -1, 0.4)
    compare(n, capi.C128, sem, every_kind(n, 500 + n, 400), start(n, n))
    compare(n, capi.C128, sem, wide, start(n, n + 1))
    compare(n, capi.C128, sem, every_kind(n, 600 + n, 150), start(n, n + 2, bad=True))


@pytest.mark.parametrize("n", [10, 16, 17, 19, 20])
def test_every_split_of_a_complex64_tile(n):
    """8 amplitudes a thread in tiles of 2^10 and 2^11, and 16."""
    compare(n, capi.C64, capi.PHYSICAL, every_kind(n, 700 + n, 400), start(n, n))
    compare(n, capi.C64, capi.PHYSICAL, every_kind(n, 800 + n, 150), start(n, n + 2, bad=True))
