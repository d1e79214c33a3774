"""The shared-tile solver at the shared-memory default: tiles whose dynamic part lies just below,
at and just above 48 KB (128 rows in 4 blocks are 48 KB to the byte) launch and match the oracle."""
import numpy as np
import pytest

from gatt_dns_b200 import case as cs

pytestmark = pytest.mark.gpu

TOL = 1e-12  # one line solve, as the other solvers are held to


@pytest.mark.parametrize("n", [124, 128, 132])
def test_tile_solver_around_48_kb(cuda_lib, oracle_lib, monkeypatch, n):
    from gatt_dns_b200.solver import GattDNS
    from oracle import Oracle
    monkeypatch.setenv("GATT_SWEEP", "tile")
    for d, shape in ((1, (n, 12, 12)), (2, (12, n, 12))):
        c = cs.periodic_box(nxyz=shape)
        f = cs.random_flow(c, seed=5)
        o, g = Oracle(c), GattDNS(c)
        for kind in ("deriv", "filter"):
            a, b = g.calc_derivs(f["U"], d, kind), o.calc_derivs(f["U"], d, kind)
            assert float(np.max(np.abs(a - b))) <= TOL * float(np.max(np.abs(b))), (d, kind)
        g.close()


def test_autotune_of_128_rows(cuda_lib):
    from gatt_dns_b200.solver import GattDNS
    g = GattDNS(cs.periodic_box(nxyz=(128, 16, 16)))
    assert g.autotune(reps=1)
    g.close()
