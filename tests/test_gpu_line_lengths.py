"""The any-length line solver at the ends of its ranges: the longest lines that tiles of 32, 16, 8 and
4 lines take, and one row more; a width asked for (GATT_LINES) that does not fit gives way."""
import functools

import numpy as np
import pytest

from gatt_dns_b200 import case as cs

pytestmark = pytest.mark.gpu

TOL = 1e-12  # one line solve, as the other solvers are held to


@functools.lru_cache(maxsize=None)
def problem(shape):
    from oracle import Oracle
    c = cs.lid_driven(nxy=shape)
    f = cs.random_flow(c, seed=4)["U"]
    d = 1 if shape[0] > shape[1] else 2
    o = Oracle(c)
    return c, f, d, {k: o.calc_derivs(f, d, k) for k in ("deriv", "filter")}


# 24, 32, 40, 48, 64, 80 and 96 blocks of 16 rows
@pytest.mark.parametrize("rows", [r + e for r in (384, 512, 640, 768, 1024, 1280, 1536) for e in (0, 1)])
@pytest.mark.parametrize("lines", ["", "8", "16", "32"])
def test_longest_lines_match_oracle(cuda_lib, oracle_lib, monkeypatch, rows, lines):
    from gatt_dns_b200.solver import GattDNS
    monkeypatch.setenv("GATT_SWEEP", "line")
    if lines:
        monkeypatch.setenv("GATT_LINES", lines)
    for shape in ((rows, 13), (13, rows)):
        c, f, d, want = problem(shape)
        with GattDNS(c) as g:
            for kind in want:
                got = g.calc_derivs(f, d, kind)
                assert np.max(np.abs(got - want[kind])) < TOL * np.max(np.abs(want[kind])), (shape, kind)
