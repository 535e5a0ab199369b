"""The calls whose speed this repository cares about, with their inputs, results and error bounds.

Every case is a whole call sequence of a user's program through the Python mirror of the C ABI: a forward
modelling run with its seismograms read back, an FWI gradient (forward with snapshots, data residual, adjoint,
assembly), or a closed-loop pass of the request server.  Grids, orders and acquisitions are those of the
benchmark's configurations and of its serving mix (NX 300-3000, NZ 150-1000, FDORDER 2-12, L 0-3, 1-16 shots);
the number of time steps is shortened so that a pass takes well under two seconds.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "denise-black-edition_b200")
_OWN = os.path.join(os.getcwd(), "denise-black-edition_b200")
sys.path.insert(0, _OWN if os.path.isdir(_OWN) else _PKG)

FL = (2.0, 8.0, 25.0)   # relaxation frequencies (Hz) of the viscoelastic runs
FW = 20                 # CPML width in points


def _case(name, **kw):
    base = dict(kind="forward", nx=600, ny=300, nt=1000, dh=5.0, dt=4e-4, fdorder=8, L=0, shots=1, own_models=False,
                nrec=120, free_surf=1, seismo=1, src_type=1, dtinv=2, snap="f32", acc="f32", ckpt=0, eprecond=0)
    base.update(kw)
    if name:
        base["name"] = name
    return base


def listed():
    return [
        # the smallest grid of the serving mix, low order: bound by launches and latency
        _case("forward_el_300x150_fd4", nx=300, ny=150, nt=2000, fdorder=4, nrec=50),
        # the plain one-shot elastic forward run of the benchmark (600 x 300, 120 receivers)
        _case("forward_el_600x300", nx=600, ny=300, nt=2000),
        # one viscoelastic shot of the benchmark's grid: an interactive single-shot run
        _case("forward_visco_2000x600", nx=2000, ny=600, nt=400, L=3, nrec=400),
        # a batch of viscoelastic shots, each on its own model (the headline batch, 16 of its 64 shots)
        _case("forward_visco_16x2000x600", nx=2000, ny=600, nt=250, L=3, shots=16, own_models=True, nrec=400),
        # an elastic survey: all shots of one line on one model (observed data, step-length tests)
        _case("forward_el_16x2000x600", nx=2000, ny=600, nt=400, shots=16, nrec=400),
        # odd sizes, the longest stencil, absorbing frame on all four sides, rotated forces, all sections
        _case("forward_el_3x1501x747_fd12", nx=1501, ny=747, nt=400, fdorder=12, shots=3, nrec=301, free_surf=0,
              seismo=4, src_type=4),
        # FWI gradient of one batch of the benchmark's gradient workload (FP16 snapshots every 2 steps)
        _case("gradient_el_8x1700x500_f16", kind="gradient", nx=1700, ny=500, nt=300, dh=10.0, dt=1e-3, shots=8,
              nrec=400, snap="f16"),
        # a small FWI: FP32 snapshots, energy preconditioning, odd sizes
        _case("gradient_el_4x601x301_f32", kind="gradient", nx=601, ny=301, nt=500, shots=4, dtinv=4, snap="f32",
              eprecond=1),
        # viscoelastic FWI with BF16 snapshots and FP64 accumulation
        _case("gradient_visco_4x1000x400_bf16", kind="gradient", nx=1000, ny=400, nt=300, L=3, shots=4, nrec=200,
              snap="bf16", acc="f64"),
        # the large-grid FWI: checkpointed adjoint with FP16 snapshots every 4 steps
        _case("gradient_el_8000x2000_ckpt", kind="gradient", nx=8000, ny=2000, nt=96, dh=2.5, dt=2e-4, nrec=1600,
              dtinv=4, snap="f16", ckpt=32),
        # the request server: a closed loop of mixed requests (elastic and viscoelastic forward, gradients)
        _case("serve_mix", kind="serve", nx=3000, ny=1000, nt=400, shots=8, nrec=300),
    ]


def draw(rng):
    """A case of the same ranges: any kind, odd sizes among them, at most the listed cases' work."""
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["forward", "forward", "forward", "gradient", "gradient", "serve"])
    if kind == "serve":
        return _case(None, kind="serve", nx=log(600, 3000), ny=log(200, 1000), nt=log(150, 400), shots=rng.randint(4, 8),
                     nrec=log(50, 300))
    nx, ny = log(300, 3000), log(150, 1000)
    L = rng.choice([0, 0, 0, 1, 2, 3])
    shots = rng.choice([1, 1, 2, 4, 8, 16])
    while shots > 1 and shots * nx * ny > (8e6 if kind == "gradient" else 2e7):
        shots //= 2
    steps = 4.0e9 / (shots * nx * ny * (2.0 if L else 1.0) * (2.5 if kind == "gradient" else 1.0))
    c = dict(kind=kind, nx=nx, ny=ny, nt=max(100, min(1500, log(300, 1500), int(steps))), L=L, shots=shots,
             fdorder=rng.choice([2, 4, 6, 8, 8, 10, 12]), nrec=log(50, 500), free_surf=rng.choice([0, 1, 1]),
             own_models=rng.random() < 0.3, src_type=rng.choice([1, 1, 2, 3, 4]))
    if kind == "gradient":
        c.update(dtinv=rng.choice([1, 2, 3, 4]), snap=rng.choice(["f32", "f16", "f16", "bf16"]),
                 acc=rng.choice(["f32", "f32", "f64"]), own_models=False, eprecond=rng.choice([0, 0, 1]))
    else:
        c.update(seismo=rng.choice([1, 1, 2, 3, 4]))
    return _case(None, **c)


# ---------------------------------------------------------------------------
# inputs (numpy only; the same arrays feed run() and exact())
# ---------------------------------------------------------------------------
def _model(nx, ny, dh, rng):
    """Velocity gradient, six layer jumps and smooth 5 % perturbations; vs and density follow vp (Gardner)."""
    z = np.arange(ny) / max(ny - 1, 1)
    v = 1800.0 + 2700.0 * z
    for d, j in zip(rng.uniform(0, 1, 6), rng.uniform(-300, 300, 6)):
        v = v + np.where(z >= d, j, 0.0)
    pert = np.zeros((nx, ny), np.float32)
    x = np.arange(nx, dtype=np.float32)[:, None]
    zz = np.arange(ny, dtype=np.float32)[None, :]
    for _ in range(3):   # separable waves of 30 to 200 cells stand for the smoothed noise
        kx, kz = 2 * np.pi / rng.uniform(30, 200, 2)
        pert += np.sin(kx * x + rng.uniform(0, 6.28)).astype(np.float32) * np.cos(kz * zz + rng.uniform(0, 6.28)).astype(np.float32)
    vp = (v[None, :].astype(np.float32) * (1 + 0.05 / 3 * pert)).astype(np.float32)
    return vp, np.maximum(vp / np.float32(1.73), np.float32(1000.0)), (310.0 * np.sqrt(np.sqrt(vp))).astype(np.float32)


def _ricker(nt, dt, fc):
    t = np.arange(1, nt + 1) * dt
    tau = np.pi * (t - 1.5 / fc) / (1.5 / fc)
    return ((1 - 4 * tau * tau) * np.exp(-2 * tau * tau)).astype(np.float32)


def _freq(c):
    """Source frequency such that the wavelet is over within the run and stays on the grid (>= 8 points per wavelength)."""
    return float(min(1000.0 / (8 * c["dh"]), max(8.0, 4.0 / (c["nt"] * c["dt"]))))


def _inputs(c, seed):
    rng = np.random.default_rng([seed, c["nx"], c["ny"], c["fdorder"]])
    nx, ny, S = c["nx"], c["ny"], c["shots"]
    models = [_model(nx, ny, c["dh"], rng) for _ in range(S if c["own_models"] else 1)]
    fc = _freq(c)
    sig = _ricker(c["nt"], c["dt"], fc)[None, :]
    shots = []
    for k in range(S):
        si = int(0.15 * nx + 0.7 * nx * (k + rng.uniform(0.2, 0.8)) / S) + 1
        n = min(c["nrec"], nx - 2 * FW - 2)
        ri = np.unique(np.linspace(FW + 1, nx - FW, n).round().astype(np.int32))
        rj = np.full(len(ri), max(2, int(round(20.0 / c["dh"]))), np.int32)
        # and a quarter as many down a borehole beside the source
        hole = np.unique(np.linspace(rj[0] + 2, ny - 2, n // 4).round().astype(np.int32))
        ri, rj = np.concatenate([ri, np.full(len(hole), min(si + 12, nx - 2), np.int32)]), np.concatenate([rj, hole])
        sj = np.array([max(2, int(round(10.0 / c["dh"])))], np.int32)
        st, az = np.array([c["src_type"]], np.int32), np.array([30.0], np.float32)
        obs = []
        if c["kind"] == "gradient":   # recorded data: a direct arrival and a later one at every receiver
            r = np.hypot(ri - si, rj)[:, None] * c["dh"] + 50.0
            t = np.arange(1, c["nt"] + 1)[None, :] * c["dt"]
            for amp in (1.0, 0.7):
                o = np.zeros((len(ri), c["nt"]))
                for v, a in ((2000.0, 1e-5), (1400.0, 6e-6)):
                    tau = np.pi * (t - 1.5 / fc - r / v) * fc / 1.5
                    o += amp * a * np.sqrt(50.0 / r) * (1 - 4 * tau * tau) * np.exp(-2 * tau * tau)
                obs.append(o.astype(np.float32))
        shots.append(dict(si=np.array([si], np.int32), sj=sj, sig=sig, ri=ri, rj=rj, st=st, az=az, obs=obs))
    return models, shots


def _requests(c):
    """The server's requests: mixed sizes (down from the case's), orders, kinds and step counts."""
    out = []
    for k in range(c["shots"]):
        f = 0.1 + 0.9 * (k + 0.5) / c["shots"]
        kind, L = [("forward", 0), ("forward", 3), ("gradient", 0), ("forward", 0)][k % 4]
        r = _case(None, kind=kind, nx=max(300, int(f * c["nx"])), ny=max(150, int(f * c["ny"])), L=L,
                  nt=int(c["nt"] * (1.0 - 0.5 * ((3 * k) % 8) / 7)), fdorder=[8, 4, 8, 12][(k + k // 4) % 4],
                  shots=1 + k % 3, nrec=c["nrec"], snap="f16")
        out.append(r)
    return out


# ---------------------------------------------------------------------------
# the framework's calls
# ---------------------------------------------------------------------------
def _params(c):
    import denise_b200 as dn
    from denise_b200 import _lib

    snap = {"f32": _lib.SNAP_F32, "f16": _lib.SNAP_F16, "bf16": _lib.SNAP_BF16}[c["snap"]]
    return dn.PsvParams(nx=c["nx"], ny=c["ny"], dh=c["dh"], dt=c["dt"], nt=c["nt"], fdorder=c["fdorder"],
                        free_surf=c["free_surf"], fw=FW, L=c["L"], fl=FL[:c["L"]], ts=1.0 / 8.0, seismo=c["seismo"],
                        dtinv=c["dtinv"], eprecond=c["eprecond"], store_snapshots=1 if c["kind"] == "gradient" else 0,
                        snap_precision=snap, grad_accum=_lib.ACC_F64 if c["acc"] == "f64" else _lib.ACC_F32,
                        ckpt_steps=c["ckpt"])


def _quality(c, model):
    if not c["L"]:
        return ()
    q = np.full(model[0].shape, 30.0, np.float32)
    return q, q


def prepare(case, seed):
    import denise_b200 as dn

    if case["kind"] == "serve":
        from denise_b200 import serve

        reqs = []
        for k, c in enumerate(_requests(case)):
            models, shots = _inputs(c, seed * 64 + k)
            obs = [tuple(s["obs"]) for s in shots] if c["kind"] == "gradient" else None
            reqs.append(serve.Request(c["kind"], _params(c), tuple(models[0]) + _quality(c, models[0]),
                                      [(s["si"], s["sj"], s["sig"], s["ri"], s["rj"]) for s in shots], obs, rid=k))
        return {"case": case, "requests": reqs}
    models, shots = _inputs(case, seed)
    p = _params(case)
    ms = [dn.Model(p, *m, *_quality(case, m)) for m in models]
    ss = [dn.Shot(ms[k % len(ms)], s["si"], s["sj"], s["sig"], s["ri"], s["rj"], src_type=s["st"], src_azi=s["az"])
          for k, s in enumerate(shots)]
    return {"case": case, "models": ms, "shots": ss, "obs": [s["obs"] for s in shots]}


def _components(c):
    return {1: (0, 1), 2: (2,), 3: (3, 4), 4: (0, 1, 2, 3, 4)}[c["seismo"]]


def run(state):
    import denise_b200 as dn

    c = state["case"]
    if c["kind"] == "serve":
        from denise_b200 import serve

        srv = serve.Server()
        for r in state["requests"]:
            srv.submit(r)
        done = {r.rid: r for r in srv.run()}
        srv.close()
        # the sections of a request's first and last shot, or its gradient and misfit
        return [[done[k].misfit, *done[k].gradient] if done[k].kind == "gradient" else
                [s[q] for s in (done[k].sections[0], done[k].sections[-1]) for q in ("vx", "vy")] for k in sorted(done)]
    shots = state["shots"]
    if c["kind"] == "forward":
        dn.run(shots, dn.MODE_FORWARD)
        return [np.stack([s.sections(q) for s in shots]) for q in _components(c)]
    m = state["models"][0]
    m.zero_gradient()
    dn.run(shots, dn.MODE_FORWARD)
    misfit = 0.0
    for s, obs in zip(shots, state["obs"]):
        misfit += s.residual(obs[0], 0) + s.residual(obs[1], 1)
    dn.run(shots, dn.MODE_ADJOINT)
    for s in shots:
        if c["eprecond"]:
            s.accumulate_gradient_precond(3000.0, 1700.0, 2200.0)
        else:
            s.accumulate_gradient()
    return [misfit, *m.gradient()]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _work(c):
    n, L = c["nx"] * c["ny"], c["L"]
    models = c["shots"] if c["own_models"] else 1
    state, mats = 5 + 3 * L, (8 if L else 5)
    # a time step reads the fields and memory variables it advances once and writes them once, and reads each
    # model's coefficients once; seismograms go out once
    step = 4.0 * n * (2 * state * c["shots"] + mats * models)
    flops = n * c["shots"] * (8.0 * (3 * c["fdorder"] // 2 - 1) + 34 + 30 * L)
    b, f = step * c["nt"], flops * c["nt"]
    b += 5.0 * c["nrec"] * c["nt"] * c["shots"] * len(_components(c))
    if c["kind"] == "gradient":
        snaps, esz = math.ceil(c["nt"] / c["dtinv"]), {"f32": 4, "f16": 2, "bf16": 2}[c["snap"]]
        # the adjoint run also advances the integrated velocities; checkpoints add one forward run; a snapshot's
        # five fields go out once and come back once, and a correlation adds to three sums
        b += step * c["nt"] * (2 if c["ckpt"] else 1) + 16.0 * n * c["shots"] * c["nt"]
        f *= 3 if c["ckpt"] else 2
        b += snaps * n * c["shots"] * (10.0 * esz + 6 * (8 if c["acc"] == "f64" else 4)) + 8.0 * n * snaps
        f += 30.0 * n * c["shots"] * snaps
        b += 12.0 * n
    return b, f


def work(case):
    parts = _requests(case) if case["kind"] == "serve" else [case]
    got = [_work(c) for c in parts]
    return {"bytes": sum(b for b, _ in got), "flops": sum(f for _, f in got)}


def tolerance(case):
    """About four times the distance from the 64-bit scheme: float sums over hundreds of time steps, and for
    gradients the rounding of the stored snapshots (11 or 8 significant bits), which largely averages out."""
    if case["kind"] == "forward":
        return {"rel": 1e-5}
    snap = "f16" if case["kind"] == "serve" else case["snap"]
    return {"rel": {"f32": 1e-5, "f16": 1e-3, "bf16": 4e-3}[snap], "max": {"f32": 4e-3, "f16": 0.1, "bf16": 0.3}[snap]}


# ---------------------------------------------------------------------------
# the scheme in 64 bits, plain torch: staggered P-SV with Holberg coefficients, CPML, free surface
# ---------------------------------------------------------------------------
_HOLBERG = {2: (1.0010,), 4: (1.1382, -0.046414), 6: (1.1965, -0.078804, 0.0081781),
            8: (1.2257, -0.099537, 0.018063, -0.0026274), 10: (1.2415, -0.11231, 0.026191, -0.0064682, 0.001191),
            12: (1.2508, -0.12034, 0.032131, -0.010142, 0.0029857, -0.00066667)}


class _Scheme:
    """A batch of shots on one grid, arrays [shot, z, x] with 8 halo cells around."""

    P = 8

    def __init__(self, c, models, shots):
        self.c, self.S = c, len(shots)
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.hc = [float(np.float32(h)) for h in _HOLBERG[c["fdorder"]]]
        self.dt, self.dh, self.nx, self.ny = float(np.float32(c["dt"])), float(np.float32(c["dh"])), c["nx"], c["ny"]
        vp, vs, rho = (torch.stack([torch.from_numpy(np.ascontiguousarray(m[k].T)) for m in models]).to(self.dev).double()
                       for k in range(3))
        self.vp, self.vs, self.rho = vp, vs, rho
        right = lambda a: torch.roll(a, -1, 2)   # noqa: E731  (one rank: the far edge wraps around)
        down = lambda a: torch.roll(a, -1, 1)    # noqa: E731
        mu = rho * vs * vs
        self.rip, self.rjp = 2.0 / (rho + right(rho)), 2.0 / (rho + down(rho))
        self.mu, self.lam = mu, rho * (vp * vp - 2 * vs * vs)
        self.uip = 4.0 / (1 / mu + 1 / right(mu) + 1 / down(mu) + 1 / down(right(mu)))
        L = self.L = c["L"]
        self.nrel = []
        if L:
            tau = float(np.float32(2.0 / 30.0))
            pts = [1.0 / (2 * math.pi * f) for f in FL[:L]]
            self.eta = [self.dt / t for t in pts]
            relax = lambda w: sum((w * t) ** 2 / (1 + (w * t) ** 2) for t in pts)   # noqa: E731
            su, ss = relax(2 * math.pi * FL[0]), relax(2 * math.pi * 8.0)
            self.tau = tau
            m0, p0, ip0 = mu / (1 + su * tau), rho * vp * vp / (1 + su * tau), self.uip / (1 + su * tau)
            k = self.dt * (1 + L * tau)
            self.fip, self.f, self.g = ip0 * k, m0 * k, p0 * k
            self.dip, self.d, self.e = ip0 * tau, m0 * tau, p0 * tau   # times eta[l]
            self.bip = [1 / (1 + 0.5 * x) for x in self.eta]
            self.cip = [1 - 0.5 * x for x in self.eta]
            self.smu, self.spi = (mu / (1 + ss * tau))[:, 0], (rho * vp * vp / (1 + ss * tau))[:, 0]
        self._frames()
        ar = torch.arange(self.S, device=self.dev)
        t = lambda a: torch.tensor(a, device=self.dev)   # noqa: E731
        P = self.P
        self.src = (ar, t([int(s["sj"][0]) for s in shots]) + P - 1, t([int(s["si"][0]) for s in shots]) + P - 1)
        self.ri = torch.stack([torch.from_numpy(s["ri"].astype(np.int64)) for s in shots]).to(self.dev) + P - 1
        self.rj = torch.stack([torch.from_numpy(s["rj"].astype(np.int64)) for s in shots]).to(self.dev) + P - 1
        self.rec = (ar[:, None], self.rj, self.ri)
        self.sig = shots[0]["sig"][0].astype(np.float64)
        self.az = float(np.float32(shots[0]["az"][0] * math.pi / 180))

    def _frames(self):
        """CPML coefficients of the frame points: {half: (left or top, right or bottom)} of (a, b); K is 1."""
        fw, dh, dt = FW, self.dh, self.dt
        thick, amax = fw * dh, math.pi * 10.0
        d0 = -5.0 * 1500.0 * math.log(0.001) / (2 * thick)

        def ab(x, clamp):
            an = x / thick
            d, al = d0 * an ** 4, amax * (1 - an)
            if clamp:
                al = max(al, 0.0)
            b = math.exp(-(d + al) * dt)
            return (d * (b - 1) / (d + al) if abs(int(d)) > 0 else 0.0), b

        self.cx, self.cy = [], []
        for half in (0.0, 0.5):
            lo = [thick - dh * (i + half) for i in range(fw)]
            hi = [dh * (i + 1 + half) for i in range(fw)]
            for out, clamp in ((self.cx, True), (self.cy, False)):
                out.append([torch.tensor([ab(x, clamp) for x in s], dtype=torch.float64, device=self.dev).T for s in (lo, hi)])

    def zero(self):
        z = lambda *s: torch.zeros(s, dtype=torch.float64, device=self.dev)   # noqa: E731
        shape = (self.S, self.ny + 2 * self.P, self.nx + 2 * self.P)
        self.vx, self.vy, self.sxx, self.syy, self.sxy = (z(*shape) for _ in range(5))
        self.px, self.py = z(self.S, self.ny, self.nx), z(self.S, self.ny, self.nx)   # vxp1, vyp1
        self.r, self.p, self.q = ([z(self.S, self.ny, self.nx) for _ in range(self.L)] for _ in range(3))
        self.psx = [[z(self.S, self.ny, FW) for _ in range(2)] for _ in range(4)]
        self.psy = [[z(self.S, FW, self.nx) for _ in range(2)] for _ in range(4)]
        self.pss = [z(self.S, FW) for _ in range(2)]

    def at(self, a, dj=0, di=0):
        P = self.P
        return a[:, P + dj:P + dj + self.ny, P + di:P + di + self.nx]

    def dx(self, a, k):   # k = 1: differences (i + m, i - m + 1), k = 0: (i + m - 1, i - m)
        return sum(h * (self.at(a, 0, m + k) - self.at(a, 0, -m - 1 + k)) for m, h in enumerate(self.hc))

    def dy(self, a, k):
        return sum(h * (self.at(a, m + k, 0) - self.at(a, -m - 1 + k, 0)) for m, h in enumerate(self.hc))

    def damp_x(self, w, psi, half):
        for side in range(2):
            a, b = self.cx[half][side]
            v = w[:, :, :FW] if side == 0 else w[:, :, -FW:]
            psi[side].mul_(b).add_(a * v)
            v += psi[side]
        return w

    def damp_y(self, w, psi, half):
        for side in range(2):
            if side == 0 and self.c["free_surf"]:
                continue
            a, b = self.cy[half][side]
            v = w[:, :FW] if side == 0 else w[:, -FW:]
            psi[side].mul_(b[:, None]).add_(a[:, None] * v)
            v += psi[side]
        return w

    def step(self, n, mode, keep=False, res=None):
        """Time step n = 1..NT; mode 1: adjoint with the sources res = (vx, vy) [shot, receiver, time]."""
        c, dt, nt = self.c, self.dt, self.c["nt"]
        ax = self.damp_x(self.dx(self.sxx, 1), self.psx[0], 1) + self.damp_y(self.dy(self.sxy, 0), self.psy[1], 0)
        ay = self.damp_x(self.dx(self.sxy, 0), self.psx[1], 0) + self.damp_y(self.dy(self.syy, 1), self.psy[0], 1)
        ax *= self.rip / self.dh
        ay *= self.rjp / self.dh
        vx, vy = self.at(self.vx), self.at(self.vy)
        if mode == 1:
            self.px += dt * vx
            self.py += dt * vy
        elif keep:
            self.px, self.py = ax, ay
        vx += dt * ax
        vy += dt * ay
        if mode == 1:
            self.vx[self.rec] += res[0][:, :, n - 1]
            self.vy[self.rec] += res[1][:, :, n - 1]
        else:
            s = float(self.sig[n - 1])
            if c["src_type"] == 2:
                self.vx[self.src] += s
            if c["src_type"] == 3:
                self.vy[self.src] += s
            if c["src_type"] == 4:
                self.vx[self.src] += -math.sin(self.az) * s
                self.vy[self.src] += math.cos(self.az) * s
        dhi = 1.0 / self.dh if self.L else dt / self.dh
        vxx = self.damp_x(self.dx(self.vx, 0) * dhi, self.psx[2], 0)
        vyx = self.damp_x(self.dx(self.vy, 1) * dhi, self.psx[3], 1)
        vyy = self.damp_y(self.dy(self.vy, 0) * dhi, self.psy[2], 0)
        vxy = self.damp_y(self.dy(self.vx, 1) * dhi, self.psy[3], 1)
        sxx, syy, sxy = self.at(self.sxx), self.at(self.syy), self.at(self.sxy)
        sh, dv = vxy + vyx, vxx + vyy
        if not self.L:
            sxy += self.uip * sh
            sxx += self.lam * dv + 2 * self.mu * vxx
            syy += self.lam * dv + 2 * self.mu * vyy
        else:
            sxy += self.fip * sh
            sxx += self.g * dv - 2 * self.f * vyy
            syy += self.g * dv - 2 * self.f * vxx
            for l in range(self.L):
                for s, mv, rate in ((sxy, self.r[l], self.dip * sh), (sxx, self.p[l], self.e * dv - 2 * self.d * vyy),
                                    (syy, self.q[l], self.e * dv - 2 * self.d * vxx)):
                    s += 0.5 * dt * mv
                    mv.mul_(self.cip[l]).sub_(rate * self.eta[l]).mul_(self.bip[l])
                    s += 0.5 * dt * mv
        if mode != 1 and c["src_type"] == 1:
            a = (float(self.sig[n]) if n < nt else 0.0) - (float(self.sig[n - 2]) if n > 1 else 0.0)
            self.sxx[self.src] += a / dt
            self.syy[self.src] += a / dt
        if c["free_surf"]:
            self._surface()

    def _surface(self):
        P, dt, X = self.P, self.dt, slice(self.P, self.P + self.nx)
        self.syy[:, P, X] = 0
        for l in range(self.L):
            self.q[l][:, 0] = 0
        vxx = vyy = 0
        for m, h in enumerate(self.hc, 1):
            self.syy[:, P - m, X] = -self.syy[:, P + m, X]
            self.sxy[:, P - m, X] = -self.sxy[:, P + m - 1, X]
            vxx = vxx + h * (self.vx[:, P, P + m - 1:P + m - 1 + self.nx] - self.vx[:, P, P - m:P - m + self.nx])
            vyy = vyy + h * (self.vy[:, P + m - 1, X] - self.vy[:, P - m, X])
        vxx, vyy = vxx / self.dh, vyy / self.dh
        for side in range(2):
            a, b = self.cx[0][side]
            v = vxx[:, :FW] if side == 0 else vxx[:, -FW:]
            self.pss[side].mul_(b).add_(a * v)
            v += self.pss[side]
        sxx = self.sxx[:, P, X]
        if not self.L:
            g, f = self.lam[:, 0], 2 * self.mu[:, 0]
            sxx -= dt * (g * g / (g + f) * vxx + g * vyy)
            return
        f, g = 2 * self.smu * (1 + self.L * self.tau), self.spi * (1 + self.L * self.tau)
        sxx -= dt * (g - f) * (g - f) * vxx / g + dt * (g - f) * vyy
        de = (2 * self.smu - self.spi) * self.tau
        for l in range(self.L):
            p = self.p[l][:, 0]
            sxx -= 0.5 * dt * p
            p += self.eta[l] / (1 + 0.5 * self.eta[l]) * (de * (f / g - 1) * vxx - de * vyy)
            sxx += 0.5 * dt * p

    def record(self, comps):
        out = {}
        vx, vy, (s, j, i) = self.vx, self.vy, self.rec
        if 0 in comps:
            out[0], out[1] = vx[self.rec], vy[self.rec]
        if 2 in comps:
            out[2] = -self.sxx[self.rec] - self.syy[self.rec]
        if 3 in comps:
            d = lambda f: sum(h * f(m) for m, h in enumerate(self.hc, 1)) * self.dt / self.dh   # noqa: E731
            k = (s * 0 if self.rho.shape[0] == 1 else s, j - self.P, i - self.P)
            out[3] = (d(lambda m: vx[s, j + m, i] - vx[s, j - m + 1, i]) - d(lambda m: vy[s, j, i + m] - vy[s, j, i - m + 1])) \
                * torch.sqrt(self.vs[k] ** 2 * self.rho[k])
            out[4] = (d(lambda m: vx[s, j, i + m - 1] - vx[s, j, i - m]) + d(lambda m: vy[s, j + m - 1, i] - vy[s, j - m, i])) \
                * torch.sqrt(self.vp[k] ** 2 * self.rho[k])
        return out

    def forward(self, comps, store=False):
        self.zero()
        c, sec, snaps = self.c, {q: [] for q in comps}, []
        self.ws = 0
        for n in range(1, c["nt"] + 1):
            keep = store and (n - 1) % c["dtinv"] == 0
            self.step(n, 0, keep)
            for q, v in self.record(comps).items():
                sec[q].append(v)
            if keep:
                snaps.append([self.px, self.py] + [self.at(a).clone() for a in (self.sxx, self.syy, self.sxy)])
                if c["eprecond"]:
                    self.ws = self.ws + self.at(self.vx) ** 2 + self.at(self.vy) ** 2
        return [torch.stack(sec[q], 2) for q in comps], snaps

    def gradient(self, obs):
        """(misfit, g_vp, g_vs, g_rho): L2 residual of the integrated traces, zero-lag correlation, stacked shots."""
        c, dt = self.c, self.dt
        sec, snaps = self.forward((0, 1), True)
        res, misfit = [], 0.0
        for k in range(2):
            d = sec[k] - torch.stack([torch.from_numpy(o[k]) for o in obs]).to(self.dev).double()
            d[:, :, 0] = 0   # the first observed sample is replaced by the synthetic one
            r = torch.cumsum(d, 2) * dt
            misfit += 0.5 * float((r * r).sum())
            res.append(r.flip(2))
        self.zero()
        muss, lamss = self.mu, self.rho * self.vp ** 2 - 2 * self.mu
        wc = wu = wr = wv = 0
        for n in range(1, c["nt"] + 1):
            self.step(n, 1, res=res)
            if (c["nt"] - n) % c["dtinv"] == 0:
                rx, ry, fx, fy, fu = snaps[(c["nt"] - n) // c["dtinv"]]
                sxx, syy, sxy = self.at(self.sxx), self.at(self.syy), self.at(self.sxy)
                t = (fx + fy) * (sxx + syy)
                wr = wr + self.px * rx + self.py * ry
                wc = wc + t
                wu = wu + fu * sxy / muss ** 2 + 0.25 * t / (lamss + muss) ** 2 + 0.25 * (fx - fy) * (sxx - syy) / muss ** 2
                if c["eprecond"]:
                    wv = wv + self.at(self.vx) ** 2 + self.at(self.vy) ** 2
        lam = -dt * wc / (4 * (lamss + muss) ** 2)
        mu, rs = -dt * wu, -dt * wr
        vp, vs, rho = self.vp, self.vs, self.rho
        g = [2 * vp * rho * lam, -4 * rho * vs * lam + 2 * rho * vs * mu, (vp ** 2 - 2 * vs ** 2) * lam + vs ** 2 * mu + rs]
        if c["eprecond"]:
            we = torch.sqrt(self.ws * wv)
            we = we + 0.005 * we.amax((1, 2), keepdim=True)
            g = [a / (we * s * s) for a, s in zip(g, (3000.0, 1700.0, 2200.0))]
        return [misfit] + [a.sum(0).T.contiguous().cpu().numpy() for a in g]


def exact(case, seed):
    """What run() returns, in 64 bits."""
    if case["kind"] == "serve":
        out = []
        for k, c in enumerate(_requests(case)):
            models, shots = _inputs(c, seed * 64 + k)
            if c["kind"] == "gradient":
                out.append(_Scheme(c, models, shots).gradient([s["obs"] for s in shots]))
            else:
                ends = [shots[0], shots[-1]] if len(shots) > 1 else shots
                sec, _ = _Scheme(c, models, ends).forward((0, 1))
                out.append([sec[q][e].cpu().numpy() for e in (0, -1) for q in (0, 1)])
        return out
    models, shots = _inputs(case, seed)
    if case["kind"] == "gradient":
        return _Scheme(case, models, shots).gradient([s["obs"] for s in shots])
    sec, _ = _Scheme(case, models, shots).forward(_components(case))
    return [a.cpu().numpy() for a in sec]
