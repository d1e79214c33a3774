"""Performance cases: what programs that use this package have it compute, over the sizes they use.

A case is a dict of plain values.  ``kind`` names the workload:

* ``lid``       2-D lid-driven cavity, uniform or stretched (tanh) mesh
* ``cavity``    boundary layer over a cavity with buffer zones and SFD, 2-D (nz = 1) or 3-D
* ``layer``     3-D boundary layer over a plate, spanwise periodic, with a blowing strip
* ``box``       periodic turbulence box;  ``forced``: the same with the turbulence forcing

and ``call`` what the program does with it in one pass:

* ``step``      one ``step`` of the time loop, its max-change read on the host
* ``run``       ``steps`` steps in one ``run`` call, nothing read in between
* ``tangent``   ``jvp`` over ``steps`` steps;  ``adjoint``: ``vjp``, a checkpoint every 2 steps
* ``arnoldi``   a Krylov space of ``krylov`` vectors for ``members`` problems side by side

A time loop goes on from where it is, so a pass of ``step``, ``run``, ``tangent`` or ``adjoint``
starts at the state that the pass before it left; after ``FRESH`` steps it starts over from the
initial flow, as the next short run of a series does (coarse cavities blow up after some
hundreds of steps, with the reference's own arithmetic too).
"""
import functools
import math

import numpy as np
import torch

from gatt_dns_b200 import case as builders
from gatt_dns_b200.solver import GattDNS

KEYS = ("U", "V", "W", "R", "E")
MEAN = ("mU", "mV", "mW", "mR", "mE")


def _c(name, kind, call, nx, ny, nz, **more):
    c = dict(kind=kind, call=call, nx=nx, ny=ny, nz=nz, steps=1, members=1, krylov=0, scheme=1, mesh="uniform")
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest flows: a time loop on a coarse 2-D grid, bound by launches and latency
        _c("lid_48_step", "lid", "step", 48, 48, 1),
        # the 128^2 cavity of Re 1000 marched at a fixed dt without reading every step
        _c("lid_128_run", "lid", "run", 128, 128, 1, steps=10),
        # an odd, stretched grid under the three-stage integrator
        _c("lid_131x97_ssp", "lid", "step", 131, 97, 1, scheme=3, mesh="tanh"),
        # global stability of the 128^2 cavity: several problems in one batch
        _c("arnoldi_128_x12", "lid", "arnoldi", 128, 128, 1, steps=10, members=12, krylov=3),
        # base flow by SFD: the 800 x 300 boundary layer over a cavity
        _c("cavity_800x300", "cavity", "step", 800, 300, 1),
        # sensitivity of a smaller 2-D cavity with SFD, state and mean
        _c("tangent_cavity_320x144", "cavity", "tangent", 320, 144, 1, steps=4),
        # the same geometry in 3-D on an odd grid
        _c("cavity3d_193x75x20", "cavity", "step", 193, 75, 20),
        # transition in the 400 x 150 x 64 boundary layer
        _c("layer_400x150x64", "layer", "step", 400, 150, 64),
        # gradient of a functional of a 3-D boundary layer's end state
        _c("adjoint_200x96x32", "layer", "adjoint", 200, 96, 32, steps=4),
        # decaying turbulence: the 128^3 box, and a box no tile divides
        _c("box_128", "box", "step", 128, 128, 128),
        _c("box_90x75x54", "box", "step", 90, 75, 54),
        # forced turbulence with the sixth-order scheme
        _c("forced_64", "forced", "step", 64, 64, 64),
    ]


def _span(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(("lid", "lid", "arnoldi", "cavity", "cavity3d", "tangent", "layer", "adjoint", "box", "box",
                       "box_odd", "forced"))
    if what == "lid":
        run = rng.random() < 0.5
        return _c("", "lid", "run" if run else "step", _span(rng, 40, 320), _span(rng, 40, 320), 1,
                  steps=rng.randint(4, 16) if run else 1, scheme=rng.choice((1, 1, 3)),
                  mesh=rng.choice(("uniform", "tanh")))
    if what == "arnoldi":
        return _c("", "lid", "arnoldi", _span(rng, 48, 144), _span(rng, 48, 144), 1, steps=rng.randint(4, 12),
                  members=rng.randint(2, 16), krylov=rng.randint(2, 4))
    if what == "cavity":
        return _c("", "cavity", "step", _span(rng, 160, 800), _span(rng, 96, 300), 1)
    if what == "cavity3d":
        return _c("", "cavity", "step", _span(rng, 128, 256), _span(rng, 64, 112), _span(rng, 8, 32))
    if what == "tangent":
        return _c("", "cavity", "tangent", _span(rng, 160, 400), _span(rng, 96, 176), 1, steps=rng.randint(2, 4))
    if what == "layer":
        return _c("", "layer", "step", _span(rng, 128, 400), _span(rng, 64, 150), _span(rng, 8, 64))
    if what == "adjoint":
        return _c("", "layer", "adjoint", _span(rng, 128, 200), _span(rng, 64, 96), _span(rng, 8, 32),
                  steps=rng.randint(2, 4))
    if what == "forced":
        n = 16 * rng.randint(2, 6)
        return _c("", "forced", "step", n, n, 16 * rng.randint(2, 6))
    if what == "box_odd":
        return _c("", "box", "step", _span(rng, 30, 120), _span(rng, 30, 120), _span(rng, 30, 120))
    return _c("", "box", "step", 16 * rng.randint(2, 8), 16 * rng.randint(2, 8), 16 * rng.randint(2, 8))


# ---- inputs ------------------------------------------------------------------------------------

def _key(case):
    return tuple(case[k] for k in ("kind", "nx", "ny", "nz", "scheme", "mesh"))


@functools.lru_cache(maxsize=4)
def _built(key):
    """The mesh, coefficient arrays and boundary lists of a case: the same for every seed."""
    kind, nx, ny, nz, scheme, mesh = key
    if kind == "lid":
        c = builders.lid_driven(nxy=(nx, ny), mesh_type=mesh)
    elif kind == "cavity":
        # 40/30/40 buffer nodes of the 800 x 300 grid, in proportion
        c = builders.boundary_layer_cavity(nx, ny, nz, buffers=((nx // 20, nx // 27), (0, ny * 2 // 15)))
    elif kind == "layer":
        c = builders.boundary_layer(nx, ny, nz, buffers=((nx // 16, nx // 20), (0, ny // 10)))
        i = int(np.nonzero(c.X > 0.5)[0][0]) + 1
        c = builders.periodic_sine_strip(c, i, i + max(6, nx // 12), omega=7.0, amp=0.01)
    elif kind == "box":
        c = builders.periodic_box(nxyz=(nx, ny, nz))
    else:
        c = builders.turbulence_box(nxyz=(nx, ny, nz))
    c.time_stepping = scheme
    return c


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _noise(gen, shape):
    """Smoothed unit noise that the compact schemes resolve, (nz, ny, nx)."""
    v = torch.randn(shape, generator=gen, dtype=torch.float64, device=_dev())
    for ax in range(3):
        if shape[ax] > 2:
            for _ in range(2):
                v = 0.25 * v.roll(1, ax) + 0.5 * v + 0.25 * v.roll(-1, ax)
    return v


def _turbulence(gen, shape):
    """A random solenoidal velocity of unit rms with the spectrum k^4 exp(-2 (k/4)^2)."""
    kz, ky, kx = torch.meshgrid(*(torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=_dev()) for n in shape),
                                indexing="ij")
    k2 = (kx * kx + ky * ky + kz * kz).clamp(min=1e-30)
    amp = torch.where(k2 > 0.5, k2 * torch.exp(-k2 / 16.0), torch.zeros_like(k2))  # sqrt(E(k) / k^2), to a factor
    hat = [amp * torch.fft.fftn(torch.randn(shape, generator=gen, dtype=torch.float64, device=_dev())) for _ in range(3)]
    div = (kx * hat[0] + ky * hat[1] + kz * hat[2]) / k2
    vel = [torch.fft.ifftn(h - k * div).real for h, k in zip(hat, (kx, ky, kz))]
    rms = (sum(v.square().mean() for v in vel) / 3.0).sqrt()
    return [v / rms for v in vel]


def _flow(case, seed, amp=0.01):
    """The initial flow of a seed: {variable: (nz, ny, nx) tensor} (a Fortran array's memory order)."""
    c = _built(_key(case))
    gen = torch.Generator(device=_dev()).manual_seed(int(seed))
    shape = (c.nz, c.ny, c.nx)
    one = torch.ones(shape, dtype=torch.float64, device=_dev())
    f = {"U": 0 * one, "V": 0 * one, "W": 0 * one, "R": one.clone(), "E": c.E0 * one}
    if case["kind"] in ("box", "forced"):
        f["U"], f["V"], f["W"] = _turbulence(gen, shape)
        return f
    if case["kind"] in ("cavity", "layer"):
        x, y = np.asarray(c.X), np.asarray(c.Y)
        delta = 5.0 * np.sqrt(np.maximum(x, 1e-12) / c.Re)
        u = np.sin(0.5 * math.pi * np.clip(y[:, None] / delta[None, :], 0.0, 1.0))
        u[:, x <= 0] = 1.0
        f["U"] = torch.from_numpy(u).to(one.device).expand(shape).clone()
    for k, s in zip(KEYS, (1.0, 1.0, 1.0 if c.nz > 1 else 0.0, 0.2, 0.2 * c.E0)):
        if s:
            f[k] = f[k] + amp * s * _noise(gen, shape)
    return f


def _dt(case):
    """The fixed time step: CFL 0.5 on the largest speed that the flow reaches."""
    c = _built(_key(case))
    speed = 1.0 / c.Ma + (4.0 if case["kind"] in ("box", "forced") else 1.5)
    return 0.5 / (speed * sum(c.dxmin[:3 if c.nz > 1 else 2]))


def _host(f):
    """{variable: tensor} as Fortran-ordered host arrays (nx, ny, nz)."""
    return {k: v.cpu().numpy().T for k, v in f.items()}


def _vectors(case, seed):
    """The tangent's input or the adjoint's: one field per variable, and per mean with SFD."""
    c = _built(_key(case))
    gen = torch.Generator(device=_dev()).manual_seed(int(seed) + 77777)
    shape = (c.nz, c.ny, c.nx)
    v = {k: _noise(gen, shape) for k in KEYS + (MEAN if c.sfd_type else ())}
    if c.nz == 1:
        for k in ("W", "mW"):
            if k in v:
                v[k] = 0 * v[k]
    return v


def _krylov_start(case, seed):
    """The Arnoldi problems' base flow and initial disturbances."""
    c = _built(_key(case))
    base = _flow(case, seed)
    gen = torch.Generator(device=_dev()).manual_seed(int(seed) + 55555)
    v0 = []
    for _ in range(case["members"]):
        z = {k: torch.zeros((c.nz, c.ny, c.nx), dtype=torch.float64, device=_dev()) for k in KEYS}
        z["U"], z["V"] = _noise(gen, z["U"].shape), _noise(gen, z["U"].shape)
        v0.append(z)
    return base, v0


EPS = 1e-4    # the Arnoldi finite difference
FRESH = 100   # steps of a run before the next one starts from the initial flow


class _Device:
    """A field of the context as the CUDA array interface describes it; a tensor made from it
    keeps it, and so the context that owns the memory, alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr, False), version=2)


def prepare(case, seed):
    c = _built(_key(case))
    g = GattDNS(c, nbatch=case["members"])
    s = dict(case=case, g=g, done=0, dt=_dt(case), shape=(c.nz, c.ny, c.nx), views={},
             keys=KEYS if c.nz > 1 else ("U", "V", "R", "E"))
    if case["call"] == "arnoldi":
        base, v0 = _krylov_start(case, seed)
        s["base"], s["v0"] = _host(base), [_host(v) for v in v0]
        return s
    f = _host(_flow(case, seed))
    for b in range(case["members"]):
        g.upload(f, b)
    g.apply_bound_cond(0.0)
    s["fresh"] = {k: v.clone() for k, v in _state(s).items()}
    if case["call"] in ("tangent", "adjoint"):
        s["vec"] = _host(_vectors(case, seed))
        if c.sfd_type:
            g.upload_mean(f)
    return s


def _state(s):
    """The context's fields where they are, as tensors."""
    g, views, out = s["g"], s["views"], {}
    for k in s["keys"]:
        p = g.device_ptr(k)
        if p not in views:
            views[p] = torch.as_tensor(_Device(g, p, s["shape"]), device="cuda")
        out[k] = views[p]
    return out


def run(s):
    case, g, n = s["case"], s["g"], s["case"]["steps"]
    call = case["call"]
    if call == "arnoldi":
        return {"H": g.arnoldi(s["base"], s["v0"], case["krylov"], n, s["dt"], eps=EPS)}
    if s["done"] + n > FRESH:
        for k, v in _state(s).items():
            v.copy_(s["fresh"][k])
        torch.cuda.current_stream().synchronize()  # the context has a stream of its own
        s["done"] = 0
    t, dt = s["done"] * s["dt"], s["dt"]
    s["done"] += n
    if call == "step":
        change = g.step(t, dt)
        return dict(_state(s), change=change)
    if call == "run":
        change = g.run(n, t, dt)
        return dict(_state(s), change=change)
    if call == "tangent":
        return {"end": g.jvp(s["vec"], n, t, dt)}
    return {"start": g.vjp(s["vec"], n, t, dt, checkpoint_every=2)}


def work(case):
    """Bytes: the states (and vectors, means) read and written once.  Operations: per point and
    stage 27 (2-D: 14) line solves of about 20 operations each and about 200 pointwise ones, per
    step 15 (8) filter solves of about 35; a tangent or adjoint step does them about three times."""
    pts = case["nx"] * case["ny"] * case["nz"] * case["members"]
    d3 = case["nz"] > 1
    nv = 5 if d3 else 4
    stages = {1: 4, 2: 1, 3: 3}[case["scheme"]]
    step = stages * ((27 if d3 else 14) * 20 + 200) + (15 if d3 else 8) * 35
    steps = case["steps"]
    fields = 2 * nv
    if case["kind"] == "cavity":
        fields += 2 * nv + 1
    if case["call"] == "arnoldi":
        steps *= case["krylov"] + 1
        fields += (case["krylov"] + 1) * nv
    if case["call"] in ("tangent", "adjoint"):
        step *= 3
        fields *= 2
    return {"bytes": 8.0 * fields * pts, "flops": float(step * steps * pts)}


# ---- the same in plain 64-bit tensor algebra ------------------------------------------------------
# Every line operator as its dense matrix, from the coefficient arrays that the case hands over;
# fields are (nz, ny, nx) tensors, a box is the 1-based [i1 i2 j1 j2 k1 k2] of the boundary lists.

def _dense(A, B, C, D, R, n_rhs, periodic, N, t):
    M = np.zeros((N, N))
    for k in range(-(n_rhs - 1), n_rhs):
        np.add.at(M, (np.arange(N), (np.arange(N) + k) % N), R[:, n_rhs - 1 + k, t])
    if not periodic:
        M[0] *= B[0, t]
        for i in range(1, N):
            M[i] = (M[i] - A[i - 1, t] * M[i - 1]) * B[i, t]
        for i in range(N - 2, -1, -1):
            M[i] -= C[i, t] * M[i + 1]
        return M
    M[0] = D[:, t] @ M
    M[1] -= A[0, t] * M[0]
    M[N - 1] -= C[0, t] * M[0]
    M[1] *= B[0, t]
    for i in range(2, N):
        M[i] = (M[i] - A[i - 1, t] * M[i - 1]) * B[i - 1, t]
    for i in range(N - 2, 0, -1):
        M[i] -= C[i, t] * M[i + 1]
    return M


class _Plain:
    """One time step of a case in plain tensor algebra."""

    def __init__(self, case):
        c = self.c = _built(_key(case))
        self.dev = _dev()
        self.d3 = c.nz > 1
        self.ops = {}
        for d, m in enumerate(c.mats):
            if m is None:
                continue
            N = (c.nx, c.ny, c.nz)[d]
            types = np.asarray(m.types)  # x: (ny, nz), y: (nx, nz), z: (nx, ny)
            lines = (types.T if d < 2 else types.T).reshape(-1)
            for kind, (A, B, C, D, R, n) in enumerate(((m.A, m.B, m.C, m.D, m.R, m.nRHS),
                                                       (m.Af, m.Bf, m.Cf, m.Df, m.Rf, m.nRHSf))):
                mats = [torch.from_numpy(_dense(A, B, C, D, R, n, m.periodic, N, t).T.copy()).to(self.dev)
                        for t in range(m.nTypes)]
                idx = [torch.from_numpy(np.nonzero(lines == t + 1)[0]).to(self.dev) for t in range(m.nTypes)]
                back = torch.argsort(torch.cat(idx))
                self.ops[d, kind] = (mats, idx, back)
        self.chi = None if not c.sfd_type else torch.from_numpy(np.ascontiguousarray(c.sfd_chi.T)).to(self.dev)

    def line(self, f, d, kind=0):
        """The line operator of direction d on the last axis of the lines of f."""
        mats, idx, back = self.ops[d, kind]
        g = f if d == 0 else (f.transpose(1, 2) if d == 1 else f.permute(1, 2, 0))
        shape = g.shape
        g = g.reshape(-1, shape[-1])
        g = g @ mats[0] if len(mats) == 1 else torch.cat([g[i] @ m for i, m in zip(idx, mats)])[back]
        g = g.reshape(shape)
        return g if d == 0 else (g.transpose(1, 2) if d == 1 else g.permute(2, 0, 1))

    def rhs(self, q):
        c = self.c
        U, V, W, R, E = (q[k] for k in KEYS)
        zero = torch.zeros_like(U)
        g, Ma = c.gamma, c.Ma
        D = {k: [self.line(q[k], 0), self.line(q[k], 1), self.line(q[k], 2) if self.d3 else zero] for k in KEYS
             if self.d3 or k != "W"}
        if not self.d3:
            D["W"] = [zero, zero, zero]
        T = g * (g - 1.0) * Ma * Ma * E
        mu = (1.0 + 110.0 / c.T0) / (T + 110.0 / c.T0) * T * torch.sqrt(T)
        (ux, uy, uz), (vx, vy, vz), (wx, wy, wz) = D["U"], D["V"], D["W"]
        div = ux + vy + wz
        s = mu / c.Re
        txx, tyy, tzz = s * (2 * ux - 2 / 3 * div), s * (2 * vy - 2 / 3 * div), s * (2 * wz - 2 / 3 * div)
        txy, txz, tyz = s * (uy + vx), s * (uz + wx), s * (vz + wy)
        h = -g / c.Re / c.Pr * mu
        heat = [h * e for e in D["E"]]

        def total(a, b, e):
            r = self.line(a, 0) + self.line(b, 1)
            return r + self.line(e, 2) if self.d3 else r

        P = (g - 1) * R * E
        dP = [(g - 1) * (R * de + dr * E) for de, dr in zip(D["E"], D["R"])]
        k = {"R": -R * div - D["R"][0] * U - D["R"][1] * V - D["R"][2] * W,
             "U": -(ux * U + uy * V + uz * W) + (total(txx, txy, txz) - dP[0]) / R,
             "V": -(vx * U + vy * V + vz * W) + (total(txy, tyy, tyz) - dP[1]) / R,
             "W": -(wx * U + wy * V + wz * W) + (total(txz, tyz, tzz) - dP[2]) / R if self.d3 else zero,
             "E": -(D["E"][0] * U + D["E"][1] * V + D["E"][2] * W)
             + (-P * div + txx * ux + tyy * vy + tzz * wz + txy * (vx + uy) + txz * (wx + uz) + tyz * (wy + vz)
                - total(*heat)) / R}
        for f in c.forcings or []:  # the turbulence forcing, over the whole box
            eps, e0 = f["par"]
            N = float(U.numel())
            ET = (U * U + V * V + W * W).sum()
            for key, x in (("U", U), ("V", V), ("W", W)):
                k[key] = k[key] + 0.25 * eps * N / ET * x - 10 * eps * x.sum() / N
            k["E"] = k["E"] - 10 * eps * (E.sum() / N - e0)
        return k

    def bound(self, q, t):
        """The boundary lists, corners and disturbances, in their order."""
        c, bc = self.c, self.c.bc
        g1 = c.gamma - 1.0
        F = {k: q[k].clone() for k in KEYS}
        get = lambda k, s: F[k][s].clone()  # noqa: E731  (a copy: the boxes are written in place)
        at = lambda b: (slice(b[4] - 1, b[5]), slice(b[2] - 1, b[3]), slice(b[0] - 1, b[1]))  # noqa: E731

        def side(b, d, m):
            """The box one list row sets, moved m nodes along direction code d (1..6: xi xf yi yf zi zf)."""
            b, a = list(b), 2 * ((d - 1) // 2)
            s = m if d % 2 else -m
            b[a] += s
            b[a + 1] += s
            return at(b)

        def extrapolated(f, b, d, coef):
            return sum(float(w) * f(side(b, d, m + 1)) for m, w in enumerate(coef))

        for V in "UVWE":
            for b, v in zip(bc.ind.get(("d", V), ()), bc.val.get(V, ())):
                F[V][at(b)] = float(v)
        for b, v in zip(bc.ind.get(("d", "P"), ()), bc.val.get("P", ())):
            F["R"][at(b)] = float(v) / g1 / get("E", at(b))

        def lists(kind, coef):
            for V in "UVWE":
                for b, d in zip(bc.ind.get((kind, V), ()), bc.dirs.get((kind, V), ())):
                    F[V][at(b)] = extrapolated(lambda s: get(V, s), b, int(d), coef)
            for b, d in zip(bc.ind.get((kind, "P"), ()), bc.dirs.get((kind, "P"), ())):
                F["R"][at(b)] = extrapolated(lambda s: get("R", s) * get("E", s), b, int(d), coef) / get("E", at(b))

        lists("n", bc.neumannCoeffs)
        for b, cd, ad in zip(bc.cL, bc.cD, bc.cAdiabatic):
            dirs = [2 * a + (1 if cd[a] == 1 else 2) for a in range(3) if cd[a]]
            if ad == 1:
                F["E"][at(b)] = sum(extrapolated(lambda s: get("E", s), b, d, bc.neumannCoeffs) for d in dirs) / len(dirs)
            P = sum(extrapolated(lambda s: get("R", s) * get("E", s), b, d, bc.neumannCoeffs) for d in dirs)
            F["R"][at(b)] = P / get("E", at(b)) / len(dirs)
        lists("s", bc.neumann2Coeffs)
        for d in bc.disturbances:
            x, b = np.asarray(d["X"], dtype=np.float64), d["ind"]
            if d["type"] == "lidDrivenMovement":
                s = 2 * (x - x[0]) / (x[-1] - x[0]) - 1
                F[d["var"]][at(b)] = torch.from_numpy(d["par"][0] * (1 - s ** 18) ** 2).to(self.dev)
            else:  # periodicSine: pi and alpha are single precision in the reference
                alpha = np.float32(2.0 * float(np.float32(4.0 * math.atan(1.0))) / (x[-1] - x[0]))
                wave = d["par"][1] * np.sin(float(alpha) * (x - x[0])) * math.sin(d["par"][0] * t)
                F[d["var"]][at(b)] = get(d["var"], at(b)) + torch.from_numpy(wave).to(self.dev)
        return F

    def step(self, q0, mean, t, dt):
        c = self.c

        def stage(q, w):
            k = self.rhs(q)
            return {v: q0[v] + w * k[v] for v in KEYS}, k

        if c.time_stepping == 2:
            q, _ = stage(q0, dt)
            q = self.bound(q, t if self.d3 else t + dt)
        elif c.time_stepping == 3:
            q, k1 = stage(q0, dt)
            k2 = self.rhs(self.bound(q, t + dt))
            q = self.bound({v: q0[v] + dt * (k1[v] + k2[v]) / 4 for v in KEYS}, t + dt / 2)
            k3 = self.rhs(q)
            q = self.bound({v: q0[v] + dt * (k1[v] + k2[v] + 4 * k3[v]) / 6 for v in KEYS}, t + dt)
        else:
            q, k1 = stage(q0, dt / 2)
            q, k2 = stage(self.bound(q, t + dt / 2), dt / 2)
            q, k3 = stage(self.bound(q, t + dt / 2), dt)
            k4 = self.rhs(self.bound(q, t + dt))
            q = {v: q0[v] + dt / 6 * (k1[v] + 2 * k2[v] + 2 * k3[v] + k4[v]) for v in KEYS}
            q = self.bound(q, t + dt)
        for d in range(3 if self.d3 else 2):
            if c.filterDirections[d]:
                q = {v: self.line(q[v], d, 1) if self.d3 or v != "W" else q[v] for v in KEYS}
        if c.sfd_type:
            mean = {v: mean[v] + dt / c.sfd_delta * (q[v] - mean[v]) for v in KEYS}
            q = {v: q[v] - dt * self.chi * (q[v] - mean[v]) for v in KEYS}
        return self.bound(q, t + dt), mean


def _exact_arnoldi(case, seed):
    p, dt = _Plain(case), _dt(case)
    keys = KEYS if p.d3 else ("U", "V", "R", "E")
    base, v0 = _krylov_start(case, seed)
    pack = lambda f: torch.cat([f[k].reshape(-1) for k in keys])  # noqa: E731
    scale = EPS * math.sqrt(len(keys) * base["U"].numel())

    def end(z):
        q, at = {k: base[k].clone() for k in KEYS}, 0
        for k in keys:
            n = q[k].numel()
            q[k] = q[k] + scale * z[at:at + n].reshape(q[k].shape)
            at += n
        for i in range(case["steps"]):
            q, _ = p.step(q, None, i * dt, dt)
        return pack(q)

    m = case["krylov"]
    H = np.zeros((case["members"], m + 1, m))
    still = end(torch.zeros_like(pack(base)))
    for b, v in enumerate(v0):
        z = pack(v)
        zeta = [z / z.norm()]
        for k in range(m):
            B = (end(zeta[k]) - still) / scale
            h = [torch.dot(z, B) for z in zeta]
            B = B - sum(x * z for x, z in zip(h, zeta))
            zeta.append(B / B.norm())
            H[b, :k + 1, k] = [float(x) for x in h]
            H[b, k + 1, k] = float(B.norm())
    return {"H": H}


def exact(case, seed):
    call, dt, n = case["call"], _dt(case), case["steps"]
    if call == "arnoldi":
        return _exact_arnoldi(case, seed)
    p = _Plain(case)
    f = _flow(case, seed)
    q = p.bound(f, 0.0)
    sfd = p.c.sfd_type > 0

    def march(q, mean):
        for i in range(n):
            last, (q, mean) = q, p.step(q, mean, i * dt, dt)
        return last, q, mean

    if call in ("step", "run"):
        last, q, _ = march(q, q)
        change = [float((q[k] - last[k]).abs().max()) for k in KEYS]
        out = {k: q[k] for k in KEYS if p.d3 or k != "W"}
        out["change"] = np.array([change])
        return out
    v = _vectors(case, seed)
    start = tuple(q[k] for k in KEYS) + (tuple(f[k] for k in KEYS) if sfd else ())
    names = KEYS + (MEAN if sfd else ())

    def flat(*x):
        _, q, mean = march(dict(zip(KEYS, x[:5])), dict(zip(KEYS, x[5:])) if sfd else None)
        return tuple(q[k] for k in KEYS) + (tuple(mean[k] for k in KEYS) if sfd else ())

    if call == "tangent":
        _, d = torch.func.jvp(flat, start, tuple(v[k] for k in names))
        return {"end": {k: x.detach().cpu().numpy().T for k, x in zip(names, d)}}
    x = [s.detach().clone().requires_grad_(True) for s in start]
    y = flat(*x)
    d = torch.autograd.grad(y, x, [v[k] for k in names])
    return {"start": {k: g.cpu().numpy().T for k, g in zip(names, d)}}
