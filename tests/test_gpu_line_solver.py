"""The any-length line solver (GATT_SWEEP=line) against the oracle: line lengths around its
16-row blocks, odd grids, several matrix types, 4, 8, 16 and 32 lines per tile, blended filters."""
import numpy as np
import pytest

from gatt_dns_b200 import case as cs

pytestmark = pytest.mark.gpu

TOL = 1e-12  # one line solve, as the other solvers are held to

CASES = {
    # cyclic: one row past a block, one short of one, one and two blocks, 8 and 32 lines of one warp
    "box_33x31x17": lambda: cs.periodic_box(nxyz=(33, 31, 17)),
    "box_16x32x24": lambda: cs.periodic_box(nxyz=(16, 32, 24)),
    "box_75x13x12": lambda: cs.periodic_box(nxyz=(75, 13, 12)),
    # walled, stretched: odd lengths, several matrix types
    "lid_131x97": lambda: cs.lid_driven(nxy=(131, 97), mesh_type="tanh"),
    "lid_21x47": lambda: cs.lid_driven(nxy=(21, 47)),
    "channel_50x37x9": lambda: cs.cavity_channel(nx=50, ny=37, nz=9),
    # long lines: more blocks than the other solvers take
    "lid_1000x23": lambda: cs.lid_driven(nxy=(1000, 23)),
    "lid_23x801": lambda: cs.lid_driven(nxy=(23, 801)),
    "box_480x12x12": lambda: cs.periodic_box(nxyz=(480, 12, 12)),
}


def rel(a, b):
    s = np.max(np.abs(b))
    return float(np.max(np.abs(a - b)) / (s if s > 0 else 1.0))


@pytest.mark.parametrize("lines", ["4", "8", "16", "32"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_line_solves_match_oracle(cuda_lib, oracle_lib, monkeypatch, name, lines):
    from gatt_dns_b200.solver import GattDNS
    from oracle import Oracle
    monkeypatch.setenv("GATT_SWEEP", "line")
    monkeypatch.setenv("GATT_LINES", lines)
    c = CASES[name]()
    f = cs.random_flow(c, seed=4)
    o = Oracle(c)
    g = GattDNS(c)
    for d in (1, 2, 3) if c.is3d else (1, 2):
        for kind in ("deriv", "filter"):
            for key in ("U", "E"):
                assert rel(g.calc_derivs(f[key], d, kind), o.calc_derivs(f[key], d, kind)) < TOL, (d, kind, key)
    for blend in (-1.0, 0.3):
        g.upload(f)
        g.apply_filters(blend)
        a, b = g.download(), o.apply_filters(f, blend)
        for key in ("U", "V", "R", "E"):
            assert rel(a[key], b[key]) < TOL, (blend, key)
    assert rel(g.nseq(f)["U"], o.nseq(f)["U"]) < TOL
    g.close()
