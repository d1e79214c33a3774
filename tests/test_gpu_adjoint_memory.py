"""Where memory is short: what the adjoint keeps only to be faster gives way to what it needs, and the
recomputing form gives the same bits; the third stream's scratch field is there where z lines use it."""
import numpy as np
import pytest

from gatt_dns_b200 import case as cs

pytestmark = pytest.mark.gpu

KEYS = ("U", "V", "W", "R", "E")


def rand_vec(c, seed):
    rng = np.random.default_rng(seed)
    keys = KEYS + (tuple("m" + k for k in KEYS) if c.sfd_type else ())
    v = {k: rng.standard_normal((c.nx, c.ny, c.nz)) for k in keys}
    if not c.is3d:
        for k in ("W", "mW"):
            if k in v:
                v[k][:] = 0.0
    return v


CASES = {
    "box": lambda: cs.periodic_box(nxyz=(24, 16, 18)),
    "lid": lambda: cs.lid_driven(nxy=(30, 24)),
    "cavity2d_sfd": lambda: cs.cavity_channel(nx=24, ny=20, nz=1, sfd={"X": 0.05, "Delta": 10.0, "buffer": 6}),
    "cavity3d": lambda: cs.cavity_channel(nx=24, ny=20, nz=8, adiabatic_corners=True),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_without_kept_sets_the_same_bits(cuda_lib, monkeypatch, name):
    from gatt_dns_b200.solver import GattDNS
    c = CASES[name]()
    f = cs.random_flow(c, seed=5, amp=0.02)
    dt = 0.25 * c.cfl_dt(f["U"], f["V"], f["W"], 1.0)
    w = rand_vec(c, 9)
    out = []
    for keep in ("1", "0"):
        monkeypatch.setenv("GATT_ADJ_KEEP", keep)
        with GattDNS(c) as g:
            g.upload(f)
            g.apply_bound_cond()
            if c.sfd_type:
                g.upload_mean(f)
            out.append((g.vjp(w, 3, 0.0, dt, checkpoint_every=2), g.rhs_vjp(f, {k: w[k] for k in KEYS})))
    for a, b in zip(*out):
        for k in a:
            assert np.array_equal(a[k], b[k]), k


def test_adjoint_fits_beside_a_full_gpu(cuda_lib):
    """96 checkpoints (1 GB) of the 64^3 box beside another program's memory: first with less free than the
    kept sets would take besides, then after a short adjoint that took them."""
    import torch
    from gatt_dns_b200.solver import GattDNS
    c = cs.periodic_box(n=64)
    f = cs.random_flow(c, seed=5, amp=0.02)
    dt = 0.25 * c.cfl_dt(f["U"], f["V"], f["W"], 1.0)
    w = rand_vec(c, 9)
    kept = 81 * 8 * c.npts        # 170 MB

    def run(g, n):
        g.upload(f)
        return g.vjp(w, n, 0.0, dt, checkpoint_every=1)

    def fill(leave):
        torch.cuda.empty_cache()
        return torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")

    torch.zeros(1, device="cuda")
    with GattDNS(c) as g:
        free = torch.cuda.mem_get_info()[0]
        want = run(g, 96)  # (and every kernel is loaded)
        used = free - torch.cuda.mem_get_info()[0]
    for first in (0, 2):
        with GattDNS(c) as g:
            free = torch.cuda.mem_get_info()[0]
            if first:
                run(g, first)
            used_now = free - torch.cuda.mem_get_info()[0]
            other = fill(used - used_now - kept // 2)
            try:
                got = run(g, 96)
            finally:
                del other
                torch.cuda.empty_cache()
        for k in want:
            assert np.array_equal(got[k], want[k]), (first, k)


def test_z_lines_through_global_memory(cuda_lib, oracle_lib, monkeypatch):
    """z lines too long for the shared tile, beside the y lines: each has a scratch field."""
    from gatt_dns_b200.solver import GattDNS
    from oracle import Oracle
    monkeypatch.setenv("GATT_SWEEP", "tile")
    c = cs.periodic_box(nxyz=(12, 16, 1200))
    f = cs.random_flow(c, seed=4)
    with GattDNS(c) as g:
        got, want = g.nseq(f), Oracle(c).nseq(f)
    for k in KEYS:
        assert np.max(np.abs(got[k] - want[k])) < 1e-12 * np.max(np.abs(want[k])), k


def test_history_that_does_not_fit(cuda_lib):
    """A run whose row-a-step history does not fit is refused, and the next one starts from no history."""
    import torch
    from gatt_dns_b200 import _lib
    from gatt_dns_b200.solver import GattDNS
    c = cs.lid_driven(n=32)
    f = cs.random_flow(c, seed=5, amp=0.02)
    dt = 0.25 * c.cfl_dt(f["U"], f["V"], f["W"], 1.0)
    torch.zeros(1, device="cuda")
    with GattDNS(c) as g:
        g.upload(f)
        want = g.run(3, 0.0, dt)
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        other = torch.empty(free - (256 << 20), dtype=torch.uint8, device="cuda")
        try:
            with pytest.raises(_lib.GattError) as e:
                g.run(1 << 23, 0.0, dt)  # 336 MB of history
            assert e.value.code == 7     # GATT_ERR_NOMEM
            g.upload(f)
            assert np.array_equal(g.run(3, 0.0, dt), want)
        finally:
            del other
            torch.cuda.empty_cache()
