"""Batches of 2-D flows in the chained step: enough members for the 32-line tiles of the combined x+y
sweep, and for more tiles than one round of CTAs.  Every member has the bits of the member alone (whose
tiles are 8 lines wide), and one is held to the oracle."""
import dataclasses

import numpy as np
import pytest

from gatt_dns_b200 import case as cs
from test_gpu_chained_2d import CASES as CHAINED

pytestmark = pytest.mark.gpu

TOL = 1e-11  # three steps, as the other step tests

# 8 blocks a line; 9 and 7, the last ones ragged; cyclic lines of 6 and 5 blocks (a block alone in its
# group of four); cyclic lines of two types (no filter: its band is not the any-length solver's); three
# types, SFD and a forcing; two members, whose tiles stay 8 lines wide
CASES = {
    "lid_128_x40": (lambda: cs.lid_driven(n=128), 40),
    "lid_131x97_tanh_ssp_x16": (lambda: dataclasses.replace(cs.lid_driven(nxy=(131, 97), mesh_type="tanh"),
                                                            time_stepping=3), 16),
    "box_96x80_x24": (lambda: cs.periodic_box(nxyz=(96, 80, 1)), 24),
    "channel_x40": (lambda: dataclasses.replace(cs.cavity_channel(nx=48, ny=40, nz=1, adiabatic_corners=True),
                                                filterDirections=(0, 0, 0)), 40),
    "bl_cavity_sfd_x40": (lambda: dataclasses.replace(
        cs.boundary_layer_cavity(nx=64, ny=48, buffers=((6, 5), (0, 6))),
        forcings=[{"type": "pressureGradient", "ind": [1, 64, 1, 48, 1, 1], "par": [0.1]}]), 40),
    "lid_48_x2": (lambda: cs.lid_driven(n=48), 2),
}


def launches_of_a_step(c, monkeypatch=None):
    """Of one member; with monkeypatch on the shared-tile solver, which is not chained: a launch for each
    direction of a sweep, two for each of the filter (by fields) and two for the max-change."""
    from gatt_dns_b200.solver import GattDNS
    if monkeypatch:
        monkeypatch.setenv("GATT_SWEEP", "tile")
    f = cs.random_flow(c, seed=3, amp=0.02)
    dt = 0.1 * c.cfl_dt(f["U"], f["V"], f["W"], 1.0)
    with GattDNS(c) as g:
        g.upload(f)
        g.apply_bound_cond()
        n = g.kernel_launches()
        g.step(0.0, dt)
        n = g.kernel_launches() - n
    if monkeypatch:
        monkeypatch.delenv("GATT_SWEEP")
    return n


@pytest.mark.parametrize("name", sorted(CASES))
def test_members_have_the_bits_of_the_member_alone(cuda_lib, oracle_lib, monkeypatch, name):
    from gatt_dns_b200.solver import GattDNS
    from oracle import Oracle
    make, members = CASES[name]
    c = make()
    flows = [cs.random_flow(c, seed=10 + b, amp=0.02) for b in range(members)]
    dt = min(0.25 * c.cfl_dt(f["U"], f["V"], f["W"], 1.0) for f in flows)
    with GattDNS(c, nbatch=members) as g:
        for b, f in enumerate(flows):
            g.upload(f, b)
        g.apply_bound_cond()
        g.step(0.0, dt)
        n = g.kernel_launches()
        change = [g.step(i * dt, dt) for i in (1, 2)]
        n = g.kernel_launches() - n
        got = [g.download(b) for b in range(members)]
    check = sorted({0, 1, members // 2, members - 1})
    for b in check:
        with GattDNS(c) as g:
            g.upload(flows[b])
            g.apply_bound_cond()
            g.step(0.0, dt)
            alone = [g.step(i * dt, dt)[0] for i in (1, 2)]
            want = g.download()
        for k in want:
            assert np.array_equal(got[b][k], want[k]), (b, k)
        assert np.array_equal([x[b] for x in change], alone)
    assert n == 2 * launches_of_a_step(c) < 2 * launches_of_a_step(c, monkeypatch)
    o = Oracle(c)
    b = check[-1]
    st = o.new_state(o.apply_bound_cond(flows[b]))
    for i in range(3):
        o.step(st, i * dt, dt)
    for k in ("U", "V", "R", "E"):
        assert np.max(np.abs(got[b][k] - st[k])) / np.max(np.abs(st[k])) < TOL, k


# (the filter of channel_sfd has a band of 11: not chained)
@pytest.mark.parametrize("name", sorted(set(CHAINED) - {"channel_sfd"}))
def test_the_cases_of_the_chained_step_are_chained(cuda_lib, monkeypatch, name):
    c = CHAINED[name]()
    stages = {1: 4, 2: 1, 3: 3}[c.time_stepping]
    assert launches_of_a_step(c, monkeypatch) - launches_of_a_step(c) == 2 * stages + 1 + sum(c.filterDirections[:2])
