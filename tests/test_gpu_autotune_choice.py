"""gatt_autotune measures the solver that it names and changes no more than the choice of solver."""
import numpy as np
import pytest

from gatt_dns_b200 import case as cs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["reg", "tile", "pipe"])
def test_tuning_keeps_the_form_of_the_step(cuda_lib, monkeypatch, solver):
    """Launches of a 2-D step: the chained form has fewer, and tuning neither brings nor takes it."""
    from gatt_dns_b200.solver import GattDNS
    monkeypatch.setenv("GATT_SWEEP", solver)
    c = cs.lid_driven(n=48)
    f = cs.random_flow(c, seed=3, amp=0.02)
    dt = 0.25 * c.cfl_dt(f["U"], f["V"], f["W"], 1.0)
    launches = []
    with GattDNS(c) as g:
        for tune in (False, True):
            if tune:
                g.autotune(reps=1)
            g.upload(f)
            g.step(0.0, dt)
            n = g.kernel_launches()
            g.step(dt, dt)
            launches.append(g.kernel_launches() - n)
    assert launches[0] == launches[1], launches
    if solver == "pipe":
        assert launches[0] < 30  # chained


@pytest.mark.parametrize("n", [24, 40, 56, 72, 88, 104])
def test_tuned_family_is_the_one_that_runs(cuda_lib, monkeypatch, n):
    """Lines of 16 blocks on a small grid, which run on the any-length solver unless tuned: a set that
    the tuner gives to the tensor-copy solver has that solver's bits, not the any-length solver's."""
    from gatt_dns_b200.solver import GattDNS
    rng = np.random.default_rng(n)
    for shape, d in (((256, n), 1), ((n, 256), 2)):
        c = cs.lid_driven(nxy=shape)
        F = np.asfortranarray(rng.standard_normal((c.nx, c.ny, 1)))
        kinds = ("deriv", "filter")
        monkeypatch.setenv("GATT_SWEEP", "line")
        with GattDNS(c) as g:
            line = [g.calc_derivs(F, d, k) for k in kinds]
        monkeypatch.setenv("GATT_SWEEP", "pipe")
        with GattDNS(c) as g:
            choice = g.autotune(reps=2)
            for i, k in enumerate(kinds):
                if choice[d, i][0] == "pipe":
                    got = g.calc_derivs(F, d, k)
                    assert not np.array_equal(got, line[i]), (shape, k)
