"""Short lists of gates that leave most amplitudes alone run as sweeps where those
move less than a pass over the state does (tiles.cu), and give the same bits.

Sizes: below, at and above the lines of the rule in each precision; conditions on
qubits whose amplitudes share 32 bytes, 128 bytes and neither."""
import pytest

from qcs_gb300 import capi
from qcs_gb300 import workloads as W
from tests.test_gpu_tiles import FORMS, compare, start

pytestmark = pytest.mark.gpu


def gates(*what):
    g = W.GateList()
    for kind, t, *rest in what:
        g.add(kind, t, rest[0] if rest else -1, 0.3 if kind in W.PARAMETRIC else 0.0)
    return g


def lists(n):
    h = n - 1
    cp = [(W.CPHASE, h, h - 2), (W.CPHASE, h - 1, h - 3), (W.CPHASE, h - 2, h - 4),
          (W.CPHASE, h - 3, h - 5)]
    return {"identities": gates((W.I, 0), (W.I, h), (W.I, 1)), "one": gates((W.I, 0), cp[0]),
            "cp2": gates(*cp[:2]), "cp3": gates(*cp[:3]), "cp4": gates(*cp),
            "low": gates((W.CPHASE, 0, 1), (W.CPHASE, 2, 1), (W.CPHASE, 3, 0)),
            "cnots": gates((W.CNOT, h, h - 1), (W.CNOT, h - 2, h - 3)),
            "phases": gates((W.P, h), (W.Z, h - 1)),
            "mixed": gates((W.CNOT, h, 2), (W.I, 3), (W.CPHASE, 4, 5), (W.Z, h))}


@pytest.mark.parametrize("prec,n,name,sweeps", [
    (capi.C64, 12, "identities", 0), (capi.C64, 12, "one", 1), (capi.C64, 12, "cp2", None),
    (capi.C64, 21, "cp2", None), (capi.C64, 22, "cp2", 2), (capi.C64, 22, "cp3", None),
    (capi.C64, 23, "cp3", 3), (capi.C64, 23, "cp4", None), (capi.C64, 24, "cp4", 4),
    (capi.C64, 24, "low", None), (capi.C64, 24, "cnots", 2), (capi.C64, 24, "phases", 2),
    (capi.C64, 24, "identities", 0),
    (capi.C128, 10, "identities", 0), (capi.C128, 10, "one", 1), (capi.C128, 19, "cp2", None),
    (capi.C128, 20, "cp2", 2), (capi.C128, 20, "cp4", None), (capi.C128, 23, "cp4", 4),
    (capi.C128, 23, "phases", None), (capi.C128, 23, "cnots", None)])
def test_what_is_launched(prec, n, name, sweeps):
    """sweeps: their number, None for one pass."""
    with capi.State(n, prec) as s:
        s.profile(True)
        s.run(lists(n)[name])
        done = {k: v[0] for k, v in s.profile_read().items()}
    assert done.pop("tile", 0) == (1 if sweeps is None else 0)
    assert sum(done.values()) == (sweeps or 0)


@pytest.mark.parametrize("prec,sem", FORMS)
@pytest.mark.parametrize("n", [6, 20, 23])
def test_the_same_bits(n, prec, sem):
    for g in lists(n).values():
        compare(n, prec, sem, g, start(n, n))
