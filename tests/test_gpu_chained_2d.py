"""2-D steps as one chain of launches (x and y sweeps together) against the oracle: line lengths
around the 16-row blocks, the integrators, blended and one-directional filters, cyclic lines with
several matrix types, SFD and a forcing, more tiles than one round."""
import dataclasses

import numpy as np
import pytest

from gatt_dns_b200 import case as cs

pytestmark = pytest.mark.gpu

TOL = 1e-11  # three steps, as the other step tests

CASES = {
    "lid_33x48_tanh": lambda: cs.lid_driven(nxy=(33, 48), mesh_type="tanh"),
    "lid_ssp_blend": lambda: dataclasses.replace(cs.lid_driven(nxy=(64, 50)), time_stepping=3, filterCharTime=0.05),
    "lid_euler_xfilter": lambda: dataclasses.replace(cs.lid_driven(n=40), time_stepping=2, filterDirections=(1, 0, 0)),
    "channel_sfd": lambda: dataclasses.replace(
        cs.cavity_channel(nx=48, ny=40, nz=1, adiabatic_corners=True, sfd={"X": 0.05, "Delta": 10.0, "buffer": 8}),
        forcings=[{"type": "pressureGradient", "ind": [1, 48, 1, 40, 1, 1], "par": [0.1]}]),
    "lid_300x260": lambda: cs.lid_driven(nxy=(300, 260)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_chained_steps_match_oracle(cuda_lib, oracle_lib, name):
    from gatt_dns_b200.solver import GattDNS
    from oracle import Oracle
    c = CASES[name]()
    f = cs.random_flow(c, seed=3, amp=0.02)
    dt = 0.25 * c.cfl_dt(f["U"], f["V"], f["W"], 1.0)
    o = Oracle(c)
    f = o.apply_bound_cond(f)
    st = o.new_state(f)
    g = GattDNS(c)
    g.upload(f)
    for i in range(3):
        mg, mo = g.step(i * dt, dt)[0], o.step(st, i * dt, dt)
        assert np.allclose(mg, mo, rtol=1e-8, atol=1e-13), (name, i, mg, mo)
    a = g.download()
    g.close()
    for k in ("U", "V", "R", "E"):
        s = np.max(np.abs(st[k]))
        assert np.max(np.abs(a[k] - st[k])) / s < TOL, (name, k)
