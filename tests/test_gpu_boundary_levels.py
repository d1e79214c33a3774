"""The boundary program sorted into levels against the oracle, which applies the lists in order:
random overlapping boxes (thin and thick) of every list kind, corners with and without E."""
import dataclasses

import numpy as np
import pytest

from gatt_dns_b200 import case as cs

pytestmark = pytest.mark.gpu

# every value is a short chain of multiply-adds and divisions of O(1) values: a few ulps each
TOL = 1e-13
LEN = 6  # Neumann coefficients of the builders


def random_bc(case, seed, items):
    rng = np.random.default_rng(seed)
    n = (case.nx, case.ny, case.nz)
    bc = cs.BoundaryInfo(neumannCoeffs=case.bc.neumannCoeffs, neumann2Coeffs=case.bc.neumann2Coeffs)

    def box(thin=None, room=None):
        out = []
        for a in range(3):
            lo = int(rng.integers(1, n[a] + 1))
            hi = int(rng.integers(lo, n[a] + 1))
            out += [lo, hi]
        if thin is not None:  # a face along direction code `thin`, or up to two planes
            a = (thin - 1) // 2
            p = int(rng.integers(1 + (0 if thin % 2 else room), n[a] - (room if thin % 2 else 0) + 1))
            q = min(p + int(rng.integers(0, 2)), n[a] - (room if thin % 2 else 0))
            out[2 * a:2 * a + 2] = [p, q]
        return out

    dirs = [d for d in range(1, 7) if n[(d - 1) // 2] > LEN + 2]
    for _ in range(items):
        v = "UVWPE"[rng.integers(0, 5)]
        kind = "dns"[rng.integers(0, 3)]
        if kind == "d":
            row = box()
            bc.ind.setdefault(("d", v), []).append(row)
            bc.val.setdefault(v, []).append(float(rng.uniform(0.5, 1.5)))
        else:
            d = int(rng.choice(dirs))
            bc.ind.setdefault((kind, v), []).append(box(d, LEN))
            bc.dirs.setdefault((kind, v), []).append(d)
    cl, cd, ca = [], [], []
    for _ in range(4):
        use = [a for a in range(3) if n[a] > LEN + 2]
        sign = [0, 0, 0]
        row = []
        for a in range(3):
            s = int(rng.choice((-1, 1))) if a in use and (rng.random() < 0.8 or a == use[0]) else 0
            sign[a] = s
            p = int(rng.integers(1 + (LEN if s < 0 else 0), n[a] - (LEN if s > 0 else 0) + 1))
            row += [p, p if s else min(n[a], p + 2)]
        cl.append(row)
        cd.append(sign)
        ca.append(int(rng.integers(0, 2)))
    bc.ind = {k: np.array(v, dtype=np.int32).reshape(-1, 6) for k, v in bc.ind.items()}
    bc.val = {k: np.array(v) for k, v in bc.val.items()}
    bc.dirs = {k: np.array(v, dtype=np.int32) for k, v in bc.dirs.items()}
    bc.cL, bc.cD, bc.cAdiabatic = (np.array(x, dtype=np.int32) for x in (cl, cd, ca))
    return bc


@pytest.mark.parametrize("shape,items,cluster", [((24, 20, 1), 12, True), ((24, 20, 1), 60, False), ((17, 13, 11), 30, True),
                                                 ((64, 48, 40), 40, True), ((24, 20, 1), 700, True)])
def test_levels_match_the_lists_in_order(cuda_lib, oracle_lib, monkeypatch, shape, items, cluster):
    from gatt_dns_b200.solver import GattDNS
    from oracle import Oracle
    if not cluster:
        monkeypatch.setenv("GATT_BC_CLUSTER", "0")
    base = cs.lid_driven(nxy=shape[:2]) if shape[2] == 1 else cs.periodic_box(nxyz=shape)
    for seed in range(3):
        c = dataclasses.replace(base, bc=random_bc(base, seed, items))
        rng = np.random.default_rng(seed + 50)
        f = {k: np.asfortranarray(rng.uniform(0.5, 1.5, shape)) for k in ("U", "V", "W", "R", "E")}
        want = Oracle(c).apply_bound_cond(f)
        g = GattDNS(c)
        g.upload(f)
        g.apply_bound_cond()
        got = g.download()
        g.close()
        for k in want:
            ok = np.isfinite(want[k])
            assert np.array_equal(ok, np.isfinite(got[k])), k
            scale = np.maximum(np.abs(want[k][ok]), 1.0)
            assert np.max(np.abs(got[k][ok] - want[k][ok]) / scale) < TOL, (k, seed)
