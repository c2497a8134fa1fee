"""The library exports the qc_* and qcs_* functions that its headers declare, and no
other: the single-header form compiles the host layer into a program, which then
calls the library by those declarations."""
import subprocess

import pytest

from qcs_gb300 import capi


def test_every_exported_function_is_declared():
    try:
        p = subprocess.run(["nm", "-D", "--defined-only", capi.LIB_PATH], capture_output=True,
                           text=True, check=True)
    except FileNotFoundError:
        pytest.skip("no nm")
    names = {line.split()[-1] for line in p.stdout.splitlines() if line.split()[-2:-1] == ["T"]}
    ours = {n for n in names if n.startswith(("qc_", "qcs_"))}
    assert ours == set(capi.declared_symbols())
