"""Sampling of states whose amplitudes are zero, below the smallest normal
float, or both signs of ordinary ones, in lanes and groups of every mixture:
each draw lies in the middle of its amplitude's share of the mass, far from
where rounding could move it, so the index is that amplitude's exactly."""
import numpy as np
import pytest

from qcs_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [capi.C64, capi.C128])
@pytest.mark.parametrize("n", [3, 7, 10, 12, 13, 15])
def test_draws_in_the_middle_of_a_share(n, prec):
    r = np.random.default_rng(n)
    size = 1 << n
    kind = r.integers(0, 4, size)
    kind[::5] = 3
    if n >= 10:
        kind[128:640] = 0  # whole groups of zeros
        kind[700:900] = 1  # and of numbers below the normal range
    a = np.where(kind == 3, r.normal(size=size) + 1j * r.normal(size=size), 0)
    a = np.where(kind == 2, 1e-20 * (1 + 1j), a)
    a = (a / np.linalg.norm(a)).astype(np.complex64)
    a[kind == 1] = np.complex64(complex(1e-40, -3e-41))
    p = a.real.astype(np.float64) ** 2 + a.imag.astype(np.float64) ** 2
    run = np.cumsum(p)
    big = np.flatnonzero(p > 1e-9)
    pick = r.choice(big, 400)
    draws = run[pick] - 0.5 * p[pick]
    with capi.State(n, prec) as s:
        s.set_amplitudes(a.astype(np.complex128))
        got = s.sample(draws)
    # tile masses of complex64 are FP32 sums: their rounding moves a draw by
    # less than 4096 * 2^-24 of a tile; below a quarter of the share is exact
    clear = p[pick] > 4e-6 * (p.sum() if prec == capi.C64 else 0)
    assert clear.sum() > 40
    assert np.array_equal(got[clear], pick[clear])
