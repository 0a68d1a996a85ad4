"""The work that users of this package have it do, as timed cases.

A pass is what a driver does with one context: describe the shots, run the
forward time loop and either fetch the seismograms (modelling) or form the
residuals against the observed data, run the adjoint loop and reduce the
shot gradients on the device (one shot loop of an inversion iteration).
Grids, FD orders, boundary widths, wavelets and snapshot intervals are those
of the seeded workloads in ``ifos_b200.workloads``; the number of time steps
is cut so that a pass stays short (every step costs the same).

``exact`` is the same computation in 64 bits, written in plain torch.
"""
import math

import numpy as np
import torch

from ifos_b200 import workloads as W
from ifos_b200.params import ShotParams
from ifos_b200.solver import ShotSolver

# FDORDER -> (MAXRELERROR, weights): Taylor for 4 and 6, Holberg 0.1 % for 8 and 12
FD = {4: (0, [9 / 8, -1 / 24]),
      6: (0, [75 / 64, -25 / 384, 3 / 640]),
      8: (1, [1.2257, -0.099537, 0.018063, -0.0026274]),
      12: (1, [1.2508, -0.12034, 0.032131, -0.010142, 0.0029857, -0.00066667])}
PHYSICS = ("psv", "visco", "sh", "acoustic")
# state planes a step reads and writes (velocity, stress) and coefficient planes it reads (velocity, stress)
STATE = {"psv": (2, 3), "visco": (2, 12), "sh": (2, 2), "acoustic": (2, 1)}
COEFF = {"psv": (2, 3), "visco": (2, 6), "sh": (1, 2), "acoustic": (2, 1)}
NCOMP = {"psv": 5, "visco": 5, "sh": 3, "acoustic": 3}


def _case(name, physics, kind, nx, ny, nt, fd, shots=1, models=1, ntr=100, dtinv=3, snap="fp32", mu=False,
          free_surf=True):
    c = {"physics": physics, "kind": kind, "nx": nx, "ny": ny, "nt": nt, "fdorder": fd, "shots": shots,
         "models": models, "ntr": ntr, "dtinv": dtinv, "snap": snap, "mu_corrected": mu, "free_surf": free_surf}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest survey of the serving stream, modelling only: latency of a short request
        _case("forward 300x100", "psv", "forward", 300, 100, 1000, 4, dtinv=2),
        # one shot of the plain elastic inversion (400 x 160, FDORDER 4, its full NT), the drop-in form
        _case("gradient 400x160", "psv", "gradient", 400, 160, 2000, 4, dtinv=2),
        # the batched form: shots over the start model and its perturbations in one context
        _case("batch 64 400x160", "psv", "gradient", 400, 160, 400, 4, shots=64, models=5, dtinv=2, snap="fp16s",
              mu=True),
        # the batched form at FDORDER 12 (SH, whose CPML covers every order)
        _case("batch 64 sh 400x160", "sh", "gradient", 400, 160, 400, 12, shots=64, models=5, dtinv=2, snap="fp16s"),
        # ragged serving requests: an odd row count, viscoelastic, two requests of one survey grouped
        _case("gradient visco 1010x336", "visco", "gradient", 1010, 336, 300, 8, shots=2),
        # an odd column count (rows do not pair up), no free surface, pressure data
        _case("gradient acoustic 777x259", "acoustic", "gradient", 777, 259, 600, 6, dtinv=2, free_surf=False),
        # one shot of the viscoelastic inversion (2000 x 600, FDORDER 8, L=3), the drop-in form
        _case("gradient visco 2000x600", "visco", "gradient", 2000, 600, 300, 8, ntr=400),
        # the headline form: as many shots as fit, 16-bit segment snapshots
        _case("batch 6 visco 2000x600", "visco", "gradient", 2000, 600, 240, 8, shots=6, ntr=400, snap="fp16s",
              mu=True),
        # the precision grid, P-SV and SH, int16-segment and fp32 snapshots
        _case("gradient psv 4000x1200", "psv", "gradient", 4000, 1200, 200, 8, ntr=400, dtinv=20, snap="i16s",
              mu=True),
        _case("gradient sh 4000x1200", "sh", "gradient", 4000, 1200, 200, 8, ntr=400, dtinv=20),
        # the largest survey of the serving stream, modelling only
        _case("forward visco 3000x1000", "visco", "forward", 3000, 1000, 150, 8),
    ]


def _bytes_flops(case):
    ph, n = case["physics"], case["nx"] * case["ny"]
    (sv, ss), (cv, cs) = STATE[ph], COEFF[ph]
    taps = case["fdorder"] // 2
    nder = {"psv": 8, "visco": 8, "sh": 4, "acoustic": 4}[ph]
    per_f = nder * (3 * taps - 1) + {"psv": 30, "visco": 96, "sh": 8, "acoustic": 12}[ph]
    other_v = {"psv": 3, "visco": 3, "sh": 2, "acoustic": 1}[ph]  # planes the velocity reads from the stress half
    other_s = {"psv": 2, "visco": 2, "sh": 1, "acoustic": 2}[ph]
    step = 4 * n * (case["shots"] * (2 * (sv + ss) + other_v + other_s) + min(case["models"], case["shots"]) * (cv + cs))
    b, f = step * case["nt"], per_f * n * case["shots"] * case["nt"]
    if case["kind"] == "gradient":
        p1 = 0 if ph == "sh" else 2
        acc = {"psv": 3, "visco": 3, "sh": 2, "acoustic": 2}[ph]
        esz = 4 if case["snap"] == "fp32" else 2
        snaps = case["nt"] // case["dtinv"]
        b += (step + 4 * n * case["shots"] * 2 * p1) * case["nt"]
        # a snapshot is written once and read once; a correlation reads the adjoint fields and updates its sums
        b += snaps * n * case["shots"] * (2 * NCOMP[ph] * esz + 4 * (NCOMP[ph] + 2 * acc))
        f = 2 * f + snaps * n * case["shots"] * 20
    return b, f


def work(case):
    """Bytes and operations of one pass: per time step every state plane is read and written once, what
    the other half step's planes contribute is read once, and each model's coefficients are read once."""
    b, f = _bytes_flops(case)
    return {"bytes": b, "flops": f}


def draw(rng):
    """One more case of the same ranges: grids from 300 x 100 to 4000 x 1200 with odd sizes, 1 to 64
    shots, every physics, the FD orders each is used with, both kinds and every snapshot format in use."""
    most = max(_bytes_flops(c)[0] for c in listed())
    while True:
        ph = rng.choice(PHYSICS)
        nx = int(round(math.exp(rng.uniform(math.log(300), math.log(4000)))))
        ny = min(1200, max(100, int(nx / rng.uniform(2.4, 3.4))))
        fd = rng.choice({"psv": (4, 8), "visco": (4, 8), "sh": (4, 8, 12), "acoustic": (4, 6, 8)}[ph])
        shots = int(math.exp(rng.uniform(0.0, math.log(64.999)))) if rng.random() < 0.6 else 1
        dtinv = rng.choice((2, 3, 10))
        nt = dtinv * int(round(math.exp(rng.uniform(math.log(60), math.log(600))) / dtinv))
        c = _case(None, ph, "gradient" if rng.random() < 0.7 else "forward", nx, ny, nt, fd, shots=shots,
                  models=min(shots, rng.choice((1, 1, 3))), ntr=rng.choice((57, 100, 400 if nx > 900 else 100)),
                  dtinv=dtinv, snap=rng.choice(("fp32", "fp16s", "i16s")), mu=rng.random() < 0.5,
                  free_surf=rng.random() < 0.8)
        snap_bytes = NCOMP[ph] * nx * ny * shots * (nt // dtinv) * (4 if c["snap"] == "fp32" else 2)
        if _bytes_flops(c)[0] <= most and snap_bytes <= 25e9:
            return c


# ---------------------------------------------------------------------------
# inputs

def _smooth_field(rng, nx, ny, cells=20):
    """Seeded smooth random field (about unit variance, clipped at 3)."""
    g = rng.standard_normal((1, 1, ny // cells + 2, nx // cells + 2)).astype(np.float32)
    f = torch.nn.functional.interpolate(torch.from_numpy(g), size=(ny, nx), mode="bicubic", align_corners=True)
    return np.clip(f[0, 0].numpy() * 1.3, -3.0, 3.0)


def _inputs(case, seed):
    """Parameters, models, geometry, wavelets and observed data of a case."""
    ph, nx, ny = case["physics"], case["nx"], case["ny"]
    fd, (rel, coeffs) = case["fdorder"], FD[case["fdorder"]]
    rng = np.random.default_rng(seed)
    dh, fw, fc, vmin, vmax = ((1.0, 20, 40.0, 1800.0, 2800.0) if nx <= 500 else
                              (2.0, 30 if nx >= 2000 else 20, 15.0, 1500.0, 4500.0) if nx <= 3000 else
                              (2.5, 30, 10.0, 1500.0, 5500.0))
    fl, tau = W.qfit_tau(3, 20.0, 5.0, 60.0) if ph == "visco" else ([], 0.0)
    p = ShotParams(nx=nx, ny=ny, nt=case["nt"], dh=dh, fdorder=fd, maxrelerror=rel, fw=fw,
                   free_surf=int(case["free_surf"]), boundary=0, vppml=vmin, fpml=fc, npower=2.0, k_max_pml=1.0,
                   L=len(fl), fl=fl, tau=tau, f_ref=fc if fl else 0.0, wavetype=2 if ph == "sh" else 1,
                   acoustic=int(ph == "acoustic"), seismo=2 if ph == "acoustic" else 1,
                   source_type=2 if ph == "sh" else 1, adjoint_type=4 if ph == "acoustic" else 1,
                   dtinv=case["dtinv"], source_shape=1)
    base = W.layered_faulted(rng, nx, ny, 12, vmin, vmax, 3, dh)
    models = []
    for k in range(case["models"]):
        vp = (base * (1.0 + 0.03 * _smooth_field(rng, nx, ny))).astype(np.float32)
        models.append({"vp": vp, "vs": (vp / np.float32(1.73)).astype(np.float32), "rho": W.gardner_rho(vp)})
    top = max(float(m["vp"].max()) for m in models) * math.sqrt(1.0 + p.L * tau)
    p.dt = W.cfl_dt(dh, top, sum(abs(c) for c in coeffs))
    margin = fw + 5
    depth = 3 if case["free_surf"] else margin  # below the absorbing strip when there is one on top
    rec = W.receiver_rows(p, np.linspace(margin, nx - margin, case["ntr"]) * dh, np.full(case["ntr"], depth * dh))
    xs = np.sort(rng.uniform(margin, nx - margin, case["shots"]))
    shots = []
    for k in range(case["shots"]):
        src = W.source_rows(p, xs[k] * dh, depth * dh, fc=fc)
        shots.append((k % case["models"], src, W.ricker(p, src), rec))
    # observed traces: a direct and a reflected arrival with moveout, plus noise
    ntr = rec.shape[1]
    t = np.arange(1, p.nt + 1, dtype=np.float32) * np.float32(p.dt)
    scale = {"psv": 3e-9, "visco": 3e-9, "sh": 3e-8, "acoustic": 5e-3}[ph] / (dh * dh)
    obs = np.zeros((case["shots"], 3, ntr, p.nt), np.float32)
    for k, (_, src, _, _) in enumerate(shots):
        off = np.abs(rec[0] - src[0, 0])[:, None].astype(np.float32) * np.float32(dh)
        for d, (depth_m, amp) in enumerate(((0.0, 1.0), (0.5 * ny * dh, 0.3))):
            tau_ = (t[None, :] - np.sqrt(off ** 2 + 4 * depth_m ** 2) / vmin) * fc - 1.5
            a = (np.float32(np.pi) * tau_) ** 2
            for c in range(3):
                obs[k, c] += amp * scale * rng.uniform(0.5, 1.5) * (1.0 - 2.0 * a) * np.exp(-a)
    obs += (0.02 * scale) * rng.standard_normal(obs.shape, dtype=np.float32)
    return p, models, shots, obs


def prepare(case, seed):
    p, models, shots, obs = _inputs(case, seed)
    gradient = case["kind"] == "gradient"
    s = ShotSolver(p, max_shots=case["shots"], max_models=case["models"], max_rec=shots[0][3].shape[1],
                   snapshots=gradient, snap_format=case["snap"], mu_corrected=case["mu_corrected"])
    if case["shots"] > 1:
        s.set_options(tile_order=3)  # shots over one model side by side, as the autotuner chooses for batches
    for k, m in enumerate(models):
        s.upload_model(m, k)
    sums = torch.zeros((5, p.ny, p.nx), dtype=torch.float32, device="cuda") if gradient else None
    return {"solver": s, "shots": shots, "obs": obs, "sums": sums}


def run(state):
    s, shots = state["solver"], state["shots"]
    n = len(shots)
    for k, (model, src, sig, rec) in enumerate(shots):
        s.setup_shot(k, src, sig, rec, model=model)
    if state["sums"] is None:
        return {"sections": s.forward(n, store=False)}
    s.forward(n, store=True, fetch=False)
    misfit, energy = s.residual_adjoint(state["obs"], n)
    s.adjoint(None, n, fetch=False)
    s.grad_sum_device(n, state["sums"].data_ptr())
    return {"gradient": state["sums"], "misfit": misfit, "energy": energy}


# ---------------------------------------------------------------------------
# the same in 64 bits

def _profiles(p, free_surf, dev):
    """CPML factors (K, a, b) at the full and half points, per axis, over the whole axis (K = 1 and
    a = b = 0 outside the strips)."""
    thick = p.fw * p.dh
    d0 = -(p.npower + 1) * p.vppml * math.log(0.001) / (2.0 * thick)
    amax = math.pi * p.fpml
    out = []
    for n, low, clamp in ((p.nx, True, True), (p.ny, not free_surf, False)):
        axes = {}
        for half in (0, 1):
            K, a, b = np.ones(n), np.zeros(n), np.zeros(n)
            strips = [(range(1, p.fw + 1), True)] if low else []
            strips.append((range(n - p.fw + 1, n + 1), False))
            for idx, left in strips:
                for i in idx:
                    x = p.dh * (i - 1) + half * p.dh / 2.0
                    dist = thick - x if left else x - ((n - 1) * p.dh - thick)
                    d = al = 0.0
                    k = 1.0
                    if dist >= 0.0:
                        nrm = dist / thick
                        d = d0 * nrm ** p.npower
                        k = 1.0 + (p.k_max_pml - 1.0) * nrm ** p.npower
                        al = amax * (1.0 - nrm)
                    if clamp:
                        al = max(al, 0.0)
                    K[i - 1], b[i - 1] = k, math.exp(-(d / k + al) * p.dt)
                    # the profile's integer abs(): the factor is zero while |d| < 1
                    a[i - 1] = d * (b[i - 1] - 1.0) / (k * (d + k * al)) if int(d) != 0 else 0.0
            axes[half] = [torch.tensor(v, dtype=torch.float64, device=dev) for v in (K, a, b)]
        out.append(axes)
    px = {h: [v[None, None, :] for v in out[0][h]] for h in (0, 1)}
    py = {h: [v[None, :, None] for v in out[1][h]] for h in (0, 1)}
    return px, py


class _Exact:
    """The time loops in torch, all shots at once: fields (shots, ny + 2H, nx + 2H) with a zero halo."""

    def __init__(self, case, seed):
        self.case, self.ph = case, case["physics"]
        self.p, models, self.shots, self.obs = _inputs(case, seed)
        p = self.p
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.c = [float(np.float32(v)) for v in FD[p.fdorder][1]]
        self.H = len(self.c)
        self.dt, self.dh = float(np.float32(p.dt)), float(np.float32(p.dh))
        self.px, self.py = _profiles(p, p.free_surf, self.dev)
        t64 = lambda k: torch.tensor(np.stack([models[m][k] for m, *_ in self.shots]), dtype=torch.float64,  # noqa: E731
                                     device=self.dev)
        self.vp, self.vs, self.rho = t64("vp"), t64("vs"), t64("rho")
        R = self.rho
        self.rjp = 1.0 / (0.5 * (R + R.roll(-1, 1)))
        self.rip = 1.0 / (0.5 * (R + R.roll(-1, 2)))
        mu = R * self.vs ** 2
        inv = 1.0 / mu
        self.mu, self.uipjp = mu, 4.0 / (inv + inv.roll(-1, 2) + inv.roll(-1, 1) + inv.roll(-1, 2).roll(-1, 1))
        self.lam = R * (self.vp ** 2 - 2 * self.vs ** 2)
        self.gac = R * self.vp ** 2
        if p.L:
            tau, ws = float(np.float32(p.tau)), 2 * math.pi * p.f_ref
            tl = [1.0 / (2 * math.pi * f) for f in p.fl]
            s = sum((ws * t) ** 2 / (1 + (ws * t) ** 2) for t in tl)
            self.eta = [self.dt / t for t in tl]
            self.tau, self.mur = tau, mu / (1 + s * tau)
            self.pir, self.muijr = self.gac / (1 + s * tau), self.uipjp / (1 + s * tau)
        n = self.case["shots"]
        rec = self.shots[0][3]
        self.rj, self.ri = (torch.tensor(rec[k], dtype=torch.long, device=self.dev) - 1 for k in (1, 0))
        self.si = torch.tensor([int(s[1][0, 0]) - 1 for s in self.shots], device=self.dev)
        self.sj = torch.tensor([int(s[1][1, 0]) - 1 for s in self.shots], device=self.dev)
        self.sig = torch.tensor(np.stack([s[2][0] for s in self.shots]), dtype=torch.float64, device=self.dev)
        self.b = torch.arange(n, device=self.dev)

    def clear(self):
        p, n, H = self.p, self.case["shots"], self.H
        names = {"psv": "vx vy sxx syy sxy", "visco": "vx vy sxx syy sxy", "sh": "vz sxz syz", "acoustic": "vx vy sp"}
        self.f = {k: torch.zeros((n, p.ny + 2 * H, p.nx + 2 * H), dtype=torch.float64, device=self.dev)
                  for k in names[self.ph].split()}
        plane = lambda: torch.zeros((n, p.ny, p.nx), dtype=torch.float64, device=self.dev)  # noqa: E731
        self.psi = {}
        self.mem = {k: [plane() for _ in range(p.L)] for k in "rpq"} if p.L else {}
        self.p1 = [plane(), plane()]

    def inner(self, k):
        return self.f[k][:, self.H:self.H + self.p.ny, self.H:self.H + self.p.nx]

    def diff(self, k, axis, forward, zone):
        """Staggered difference along x (axis 2) or y (axis 1), through the CPML memory `zone` (half point or not)."""
        f, H, (ny, nx) = self.f[k], self.H, (self.p.ny, self.p.nx)

        def at(s):
            return f[:, H:H + ny, H + s:H + s + nx] if axis == 2 else f[:, H + s:H + s + ny, H:H + nx]

        out = 0
        for m, c in enumerate(self.c, 1):
            out = out + (at(m) - at(1 - m) if forward else at(m - 1) - at(-m)) * c
        return self.absorb(out * self.scale, axis, forward if zone is None else zone, k)

    def absorb(self, d, axis, half, key):
        K, a, b = (self.px if axis == 2 else self.py)[1 if half else 0]
        key = (key, axis, half)
        if key not in self.psi:
            self.psi[key] = torch.zeros_like(d)
        psi = self.psi[key] = b * self.psi[key] + a * d
        return d / K + psi

    def mirror(self, k, even):
        """Rows above the free surface as the velocity update sees them."""
        if not self.p.free_surf:
            return
        f, H = self.f[k], self.H
        for m in range(1, H + 1):
            f[:, H - m] = -f[:, H + m if even else H + m - 1]

    def velocity(self, adjoint):
        """The particle velocities; returns the snapshot's velocity components."""
        dt, ph, self.scale = self.dt, self.ph, 1.0
        if ph == "sh":
            self.mirror("syz", True)
            f = self.diff("sxz", 2, False, None) + self.diff("syz", 1, True, None)
            old = self.inner("vz").clone()
            self.inner("vz").add_(self.rjp * dt * f / self.dh)
            return [old]
        if ph == "acoustic":
            self.mirror("sp", True)
            fx, fy = self.diff("sp", 2, True, None), self.diff("sp", 1, True, None)
        else:
            self.mirror("syy", True)
            self.mirror("sxy", False)
            fx = self.diff("sxx", 2, True, None) + self.diff("sxy", 1, False, None)
            fy = self.diff("sxy", 2, False, None) + self.diff("syy", 1, True, None)
        if adjoint:
            self.p1[0] += self.inner("vx") * dt
            self.p1[1] += self.inner("vy") * dt
            p1 = self.p1
        else:
            p1 = [self.rip * fx / self.dh, self.rjp * fy / self.dh]
        self.inner("vx").add_(dt * self.rip * fx / self.dh)
        self.inner("vy").add_(dt * self.rjp * fy / self.dh)
        return p1

    def stress(self, source, pressure):
        """The stresses, then the explosive source (or pressure residuals) and the free surface."""
        p, dt, ph = self.p, self.dt, self.ph
        self.scale = (1.0 if p.L else dt) / self.dh
        fs = p.free_surf
        if ph == "sh":
            zx, zy = self.diff("vz", 2, True, None), self.diff("vz", 1, False, None)
            self.inner("sxz").add_(self.uipjp * zx)
            self.inner("syz").add_(self.mu * zy)
            if fs:
                self.inner("syz")[:, 0] = 0
            return
        vxx, vyy = self.diff("vx", 2, False, None), self.diff("vy", 1, False, None)
        if ph == "acoustic":
            sp = self.inner("sp")
            sp.add_(self.gac * (vxx + vyy))
            if source is not None:
                sp[self.b, self.sj, self.si] += source
            if pressure is not None:
                sp[:, self.rj, self.ri] += pressure
            if fs:
                sp[:, 0] = 0
            return
        vyx, vxy = self.diff("vy", 2, True, None), self.diff("vx", 1, True, None)
        sxx, syy, sxy = (self.inner(k) for k in ("sxx", "syy", "sxy"))
        half = dt / 2.0
        if not p.L:
            lam, mu = self.lam, self.mu
            sxy.add_(self.uipjp * (vyx + vxy))
            sxx.add_(lam * (vxx + vyy) + 2 * mu * vxx)
            syy.add_(lam * (vxx + vyy) + 2 * mu * vyy)
        else:
            L, tau = p.L, self.tau
            grow = dt * (1 + L * tau)
            g, f, fij = self.pir * grow, self.mur * grow, self.muijr * grow
            div, shear = vxx + vyy, vxy + vyx
            r, pp, q = self.mem["r"], self.mem["p"], self.mem["q"]
            sxy.add_(fij * shear + half * sum(r))
            sxx.add_(g * div - 2 * f * vyy + half * sum(pp))
            syy.add_(g * div - 2 * f * vxx + half * sum(q))
            for l in range(L):
                e = self.eta[l]
                b, c = 1.0 / (1.0 + 0.5 * e), 1.0 - 0.5 * e
                dip, d, ee = self.muijr * e * tau, self.mur * e * tau, self.pir * e * tau
                r[l] = b * (r[l] * c - dip * shear)
                pp[l] = b * (pp[l] * c - ee * div + 2 * d * vyy)
                q[l] = b * (q[l] * c - ee * div + 2 * d * vxx)
            sxy.add_(half * sum(r))
            sxx.add_(half * sum(pp))
            syy.add_(half * sum(q))
        if source is not None:
            sxx[self.b, self.sj, self.si] += 0.5 * source
            syy[self.b, self.sj, self.si] += 0.5 * source
        if fs:
            self.surface(sxx, syy)

    def surface(self, sxx, syy):
        H, p, dt = self.H, self.p, self.dt
        syy[:, 0] = 0
        vx, vy, nx = self.f["vx"][:, H], self.f["vy"], p.nx
        vxx = vyy = 0
        for m, c in enumerate(self.c, 1):
            vxx = vxx + c * (vx[:, H + m - 1:H + m - 1 + nx] - vx[:, H - m:H - m + nx])
            vyy = vyy + c * (vy[:, H + m - 1, H:H + nx] - vy[:, H - m, H:H + nx])
        vxx, vyy = (vxx / self.dh)[:, None, :], (vyy / self.dh)[:, None, :]
        vxx = self.absorb(vxx, 2, False, "surface")
        if not p.L:
            g, f = self.lam[:, :1], 2 * self.mu[:, :1]
            sxx[:, :1] += -dt * (g * g / (g + f) * vxx + g * vyy)
            return
        grow = 1 + p.L * self.tau
        mu, pi = self.mur[:, :1], self.pir[:, :1]
        f, g, d, e = 2 * mu * grow, pi * grow, 2 * mu * self.tau, pi * self.tau
        pp, half = self.mem["p"], dt / 2.0
        for q in self.mem["q"]:
            q[:, 0] = 0
        row = sxx[:, :1]
        row += -(dt * (g - f) ** 2 * vxx / g) - dt * (g - f) * vyy - half * sum(v[:, :1] for v in pp)
        for l in range(p.L):
            bjm = self.eta[l] / (1.0 + 0.5 * self.eta[l])
            pp[l][:, :1] += bjm * ((d - e) * (f / g - 1.0) * vxx - (d - e) * vyy)
        row += half * sum(v[:, :1] for v in pp)

    def source_term(self, nt):
        s, NT, dh = self.sig, self.p.nt, self.dh
        a = s[:, nt] if nt < NT else 0.0
        b = s[:, nt - 2] if nt > 1 else 0.0
        return (a - b) / (2.0 * dh * dh)

    def forward(self, store):
        p, ph, n = self.p, self.ph, self.case["shots"]
        self.clear()
        sec = torch.zeros((n, 6, len(self.ri), p.nt), dtype=torch.float64, device=self.dev)
        snaps = []
        for nt in range(1, p.nt + 1):
            p1 = self.velocity(False)
            if ph == "sh":
                amp = self.sig[:, nt - 1] / (self.dh * self.dh) * self.dt
                self.inner("vz")[self.b, self.sj, self.si] += self.rjp[self.b, self.sj, self.si] * amp
                self.stress(None, None)
            else:
                self.stress(self.source_term(nt), None)
            for k, plane in {"acoustic": (("sp", 3),), "sh": (("vz", 2),)}.get(ph, (("vx", 0), ("vy", 1))):
                v = self.inner(k)[:, self.rj, self.ri]
                sec[:, plane, :, nt - 1] = -v if plane == 3 else v
            if store and (nt - 1) % p.dtinv == 0:
                snaps.append([v.clone() for v in p1] + [self.inner(k).clone() for k in self.stored()])
        return sec, snaps

    def stored(self):
        return {"sh": ("sxz", "syz"), "acoustic": ("sp",)}.get(self.ph, ("sxx", "syy", "sxy"))

    def gradient(self):
        p, ph, n, dt = self.p, self.ph, self.case["shots"], self.dt
        sec, snaps = self.forward(True)
        planes = {"acoustic": ((2, 3),), "sh": ((2, 2),)}.get(ph, ((0, 0), (1, 1)))
        obs = torch.tensor(self.obs, dtype=torch.float64, device=self.dev)
        adj, misfit, energy = {}, 0, 0
        for k, plane in planes:
            d = obs[:, k].cumsum(-1) * dt
            r = sec[:, plane].cumsum(-1) * dt - d
            misfit, energy = misfit + (r * r).sum((1, 2)), energy + (d * d).sum((1, 2))
            adj[k] = r.flip(-1)
        del sec, obs
        self.clear()
        zero = lambda: torch.zeros((n, p.ny, p.nx), dtype=torch.float64, device=self.dev)  # noqa: E731
        wl, wm, wr, wmz, wrz = (zero() for _ in range(5))
        mm, ll = self.mu ** 2, (self.rho * self.vp ** 2 - self.mu) ** 2
        for nt in range(1, p.nt + 1):
            p1 = self.velocity(True)
            if ph == "sh":
                self.inner("vz")[:, self.rj, self.ri] += adj[2][:, :, nt - 1]
                self.stress(None, None)
            elif ph == "acoustic":
                self.stress(None, adj[2][:, :, nt - 1])
            else:
                self.inner("vx")[:, self.rj, self.ri] += adj[0][:, :, nt - 1]
                self.inner("vy")[:, self.rj, self.ri] += adj[1][:, :, nt - 1]
                self.stress(None, None)
            if (p.nt - nt) % p.dtinv:
                continue
            s = snaps.pop()
            if ph == "sh":
                wrz += p1[0] * s[0]
                wmz += (s[1] * self.inner("sxz") + s[2] * self.inner("syz")) / mm
                continue
            wr += p1[0] * s[0] + p1[1] * s[1]
            if ph == "acoustic":
                wl += s[2] * self.inner("sp")
                continue
            sxx, syy, sxy = (self.inner(k) for k in ("sxx", "syy", "sxy"))
            fx, fy, fu = s[2:]
            wl += (fx + fy) * (sxx + syy)
            if self.case["mu_corrected"]:
                plus, minus = (fx + fy) * (sxx + syy), (fx - fy) * (sxx - syy)
            else:
                plus, minus = fx + fy * (sxx + syy), fx - fy * (sxx - syy)
            wm += fu * sxy / mm + 0.25 * plus / ll + 0.25 * minus / mm
        pi, u, rho = self.vp, self.vs, self.rho
        vp = vs = dr = zero()
        vz, rz = wmz, wrz
        if ph == "sh":
            vz, rz = 2 * rho * u * (-dt * wmz), u * u * (-dt * wmz) - dt * wrz
        elif ph == "acoustic":
            lam = -dt * wl / (rho * pi * pi) ** 2
            vp, dr = 2 * pi * rho * lam, pi * pi * lam - dt * wr
        else:
            lam, mu = -dt * wl / (4 * ll), -dt * wm
            vp, vs = 2 * pi * rho * lam, -4 * rho * u * lam + 2 * rho * u * mu
            dr = (pi * pi - 2 * u * u) * lam + u * u * mu - dt * wr
        g = torch.stack([v.sum(0) for v in (vp, vs, dr, vz, rz)])
        return {"gradient": g, "misfit": misfit, "energy": energy}


def exact(case, seed):
    e = _Exact(case, seed)
    if case["kind"] == "forward":
        return {"sections": e.forward(False)[0]}
    return e.gradient()
