"""Boundary programs of many items against the oracle, applied once and in time steps: levels of up
to, and of more ops than a launch stages in shared memory, more Dirichlet values than a step's table
of classes holds, more levels than get a launch each, boxes under hundreds of others."""
import dataclasses

import numpy as np
import pytest

from gatt_dns_b200 import case as cs

pytestmark = pytest.mark.gpu

BC_TOL = 1e-13    # a value is one multiply-add chain of O(1) values
STEP_TOL = 1e-11  # two steps, as the other step tests
LEN = 6           # Neumann coefficients of the builders


def points(shape, n):
    """n grid points, every second one along x and y."""
    out = [(i, j, k) for k in range(1, shape[2] + 1) for j in range(1, shape[1] + 1, 2)
           for i in range(1, shape[0] + 1, 2)]
    assert len(out) >= n
    return [[i, i, j, j, k, k] for i, j, k in out[:n]]


def dirichlet(base, n):
    """n points of constant U and of constant pressure: 2 n independent items."""
    s = np.sin(np.arange(n))
    bc = cs.BoundaryInfo(neumannCoeffs=base.bc.neumannCoeffs, neumann2Coeffs=base.bc.neumann2Coeffs)
    box = np.array(points((base.nx, base.ny, base.nz), n), dtype=np.int32)
    p0 = (base.gamma - 1.0) * base.E0
    bc.ind = {("d", "U"): box, ("d", "P"): box}
    bc.val = {"U": 0.01 * s, "P": p0 * (1.0 + 0.001 * s)}
    return bc


def neumann(base, n):
    """n faces of one point for U and for V, none read by another: 2 n independent items."""
    bc = cs.BoundaryInfo(neumannCoeffs=base.bc.neumannCoeffs, neumann2Coeffs=base.bc.neumann2Coeffs)
    box = [[i, i, j, j, k, k] for k in range(1, base.nz + 1) for j in range(1, base.ny - LEN + 1, LEN + 2)
           for i in range(1, base.nx + 1)][:n]
    assert len(box) == n
    for v in "UV":
        bc.ind["n", v] = np.array(box, dtype=np.int32)
        bc.dirs["n", v] = np.full(n, cs.DIR_CODE["yi"], dtype=np.int32)
    return bc


def chain(base, n):
    """n columns of U, each extrapolated from the ones set before it: n levels."""
    bc = cs.BoundaryInfo(neumannCoeffs=base.bc.neumannCoeffs, neumann2Coeffs=base.bc.neumann2Coeffs)
    bc.ind["n", "U"] = np.array([[i, i, 1, base.ny, 1, base.nz] for i in range(n, 0, -1)], dtype=np.int32)
    bc.dirs["n", "U"] = np.full(n, cs.DIR_CODE["xi"], dtype=np.int32)
    return bc


LID = lambda: cs.lid_driven(nxy=(128, 96))  # noqa: E731
BOX = lambda: cs.periodic_box(nxyz=(32, 24, 40))  # noqa: E731

CASES = {
    "classes_200": (LID, dirichlet, 200),     # the step's assembly sets the values of U
    "classes_300": (LID, dirichlet, 300),     # more than 255 classes
    "level_204x2": (LID, dirichlet, 204),     # 409 ops: the most that a launch stages
    "level_205x2": (LID, dirichlet, 205),
    "level_967x2": (LID, dirichlet, 967),     # 1934: 227 KB of ops
    "level_968x2": (LID, dirichlet, 968),
    "level_3000x2": (LID, dirichlet, 3000),
    "faces_300x2": (LID, neumann, 300),
    "faces_1400x2": (LID, neumann, 1400),
    "faces_1400x2_3d": (BOX, neumann, 1400),
    "levels_16": (LID, chain, 16),            # the most that get a launch each
    "levels_17": (LID, chain, 17),
    "levels_20_3d": (BOX, chain, 20),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_many_items_match_oracle(cuda_lib, oracle_lib, name):
    from gatt_dns_b200.solver import GattDNS
    from oracle import Oracle
    base, lists, n = CASES[name]
    base = base()
    c = dataclasses.replace(base, bc=lists(base, n))
    f = cs.random_flow(c, seed=3, amp=0.02)
    o, g = Oracle(c), GattDNS(c)
    g.upload(f)
    g.apply_bound_cond()
    got, want = g.download(), o.apply_bound_cond(f)
    for k in want:
        assert np.max(np.abs(got[k] - want[k]) / np.maximum(np.abs(want[k]), 1.0)) < BC_TOL, k
    dt = 0.1 * c.cfl_dt(f["U"], f["V"], f["W"], 1.0)
    st = o.new_state(want)
    g.upload(want)
    for i in range(2):
        mg, mo = g.step(i * dt, dt)[0], o.step(st, i * dt, dt)
        assert np.allclose(mg, mo, rtol=1e-8, atol=1e-13), (i, mg, mo)
    got = g.download()
    g.close()
    for k in ("U", "V", "R", "E"):
        assert np.max(np.abs(got[k] - st[k])) / np.max(np.abs(st[k])) < STEP_TOL, k


def covered(base, n, lists):
    """A box over the whole grid and n small overlapping ones in each of the lists."""
    rng = np.random.default_rng(n)
    shape = (base.nx, base.ny, base.nz)
    bc = cs.BoundaryInfo(neumannCoeffs=base.bc.neumannCoeffs, neumann2Coeffs=base.bc.neumann2Coeffs)
    ref = {"U": 0.1, "E": base.E0, "P": (base.gamma - 1.0) * base.E0}
    for v in "UEP":
        m = n if v in lists else 0
        lo = rng.integers(1, np.array(shape) + 1, size=(m, 3))
        hi = np.minimum(lo + rng.integers(0, 6, size=(m, 3)), shape)
        small = np.stack([lo[:, 0], hi[:, 0], lo[:, 1], hi[:, 1], lo[:, 2], hi[:, 2]], axis=1)
        bc.ind["d", v] = np.concatenate([[[1, shape[0], 1, shape[1], 1, shape[2]]], small]).astype(np.int32)
        bc.val[v] = ref[v] * (1.0 + 0.01 * (np.arange(m + 1) % 3))
    return bc


# The large box comes apart into up to ten pieces for each small one: as pieces the 4503 boxes of the
# 3-D "UEP" program took 20 s to prepare and 9.2 ms to apply; as they are 0.07 s and 0.8 ms.
@pytest.mark.parametrize("shape", [(128, 96, 1), (48, 40, 44)])
@pytest.mark.parametrize("lists", ["U", "E", "P", "EP", "UEP"])
def test_large_box_under_small_ones(cuda_lib, oracle_lib, shape, lists):
    import time
    from gatt_dns_b200.solver import GattDNS
    from oracle import Oracle
    base = cs.lid_driven(nxy=shape[:2]) if shape[2] == 1 else cs.periodic_box(nxyz=shape)
    c = dataclasses.replace(base, bc=covered(base, 1500, lists))
    f = cs.random_flow(c, seed=3, amp=0.02)
    o, g = Oracle(c), GattDNS(c)
    g.upload(f)
    t = time.perf_counter()
    g.apply_bound_cond()
    assert time.perf_counter() - t < 1.0
    got, want = g.download(), o.apply_bound_cond(f)
    for k in want:
        assert np.max(np.abs(got[k] - want[k]) / np.maximum(np.abs(want[k]), 1.0)) < BC_TOL, k
    dt = 0.1 * c.cfl_dt(f["U"], f["V"], f["W"], 1.0)
    st = o.new_state(want)
    g.upload(want)
    mg, mo = g.step(0.0, dt)[0], o.step(st, 0.0, dt)
    assert np.allclose(mg, mo, rtol=1e-8, atol=1e-13), (mg, mo)
    got = g.download()
    g.close()
    for k in ("U", "V", "R", "E"):
        assert np.max(np.abs(got[k] - st[k])) / np.max(np.abs(st[k])) < STEP_TOL, k
