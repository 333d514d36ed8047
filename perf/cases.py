"""The work that programs of this framework have it do, as cases that can be timed and checked.

Every case is one pass of a user's program through the public classes: the initial state goes in from host arrays, the
model steps (or the network runs), and the result comes back as host arrays. `listed` names the cases, `draw` makes
more of the same ranges, `prepare` builds what the program holds before the call (an engine and its inputs), `run` is
the pass, `work` counts what it cannot do without, and `exact` is the same pass in 64 bits with torch alone.
"""
from __future__ import annotations

import math
from functools import lru_cache

import numpy as np
import torch

import lmweather_gb300 as lw

A, OMEGA, G = 6.37122e6, 7.292e-5, 9.80616  # Earth: radius (m), rotation (1/s), gravity (m/s^2)
PRECISION = {"fp64": dict(precision=lw.FP64), "fp32": dict(precision=lw.FP32),
             "split3": dict(precision=lw.SPLIT_BF16, split_terms=3), "split6": dict(precision=lw.SPLIT_BF16, split_terms=6)}


def _sphere(name, truncation, precision, members, steps, tracer=False, mountain=False, tilt=0.0):
    return {"name": name, "kind": "sphere", "truncation": truncation, "precision": precision, "members": members, "steps": steps,
            "tracer": tracer, "mountain": mountain, "tilt": tilt}


def _plane(name, nx, ny, steps, viscosity=0.0, drag=0.0, linear=False):
    return {"name": name, "kind": "plane", "nx": nx, "ny": ny, "steps": steps, "viscosity": viscosity, "drag": drag, "linear": linear}


def _mlp(name, kind, features, hidden, batch):
    return {"name": name, "kind": kind, "features": features, "hidden": hidden, "batch": batch}


def listed():
    return [
        # a script that steps the smallest model by hand and looks at the state after each step: latency and launches
        _sphere("t21_fp64_step", 21, "fp64", 1, 1),
        # the reference's own run, T42 at 900 s, 64 steps between looks at the state
        _sphere("t42_fp64_run", 42, "fp64", 1, 64),
        # a truncation between the usual ones, three members with a passive tracer over a mountain
        _sphere("t31_fp64_tracer", 31, "fp64", 3, 24, tracer=True, mountain=True),
        # high resolution in the parity precision
        _sphere("t170_fp64_run", 170, "fp64", 1, 16),
        # a few members in single precision
        _sphere("t63_fp32_members", 63, "fp32", 5, 32),
        # high resolution in the split precision, one member
        _sphere("t170_split3_run", 170, "split3", 1, 32),
        # eighteen members (two member tiles, the second nearly empty) in the six-product split precision
        _sphere("t106_split6_members", 106, "split6", 18, 16),
        # the benchmark's forecast ensemble: 1024 members of mixed truncations, rotation rates and depths in the split
        # precision, six model hours between state exchanges
        {"name": "ensemble_split3", "kind": "ensemble", "t21": 512, "t42": 384, "t85": 128, "precision": "split3", "hours": 6.0},
        # the channel model at the size of the reference's scripts
        _plane("plane_60x30", 60, 30, 100),
        # the channel model at its benchmark size
        _plane("plane_1024x512", 1024, 512, 64),
        # inference with the surrogate network of T42 states (5676 features, hidden width 4096)
        _mlp("mlp_forward", "forward", 5676, 4096, 512),
        # one training step of a T21 network: loss, gradients, Adam, and the new weights
        _mlp("mlp_train", "train", 1518, 1024, 256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sphere"] * 6 + ["ensemble", "plane", "plane", "forward", "train"])
    if kind == "sphere":
        precision = rng.choice(["fp64", "fp64", "fp32", "split3", "split6"])
        T, B = _log(rng, 21, 170), _log(rng, 1, 20)
        # the cost of a pass grows as T^3 times members and steps; FP64 steps cost about four times the others
        steps = max(1, min(_log(rng, 1, 64), int((8e7 if precision == "fp64" else 3e8) / (T ** 3 * B))))
        c = _sphere("", T, precision, B, steps, tracer=precision == "fp64" and rng.random() < 0.25, mountain=rng.random() < 0.25,
                    tilt=rng.choice([0.0, 0.0, 0.0, round(rng.uniform(0.02, 1.5), 2)]))
    elif kind == "ensemble":
        n = _log(rng, 8, 96)
        c = {"kind": "ensemble", "t21": 4 * n + rng.randrange(4), "t42": 3 * n - rng.randrange(3), "t85": n + rng.randrange(3) - 1,
             "precision": rng.choice(["split3", "split3", "split6", "fp32"]), "hours": round(rng.uniform(1.0, 5.5), 2)}
    elif kind == "plane":
        nx, ny = _log(rng, 40, 1024), _log(rng, 20, 512)
        c = _plane("", nx, ny, max(2, min(_log(rng, 8, 128), int(3.3e7 / (nx * ny)))), viscosity=rng.choice([0.0, 0.0, 50.0]),
                   drag=rng.choice([0.0, 1e-6]), linear=rng.random() < 0.2)
    else:
        T = rng.randrange(21, 43)
        c = _mlp("", kind, 3 * (T + 1) * (T + 2), 128 * _log(rng, 4, 32 if kind == "forward" else 8), 128 * rng.randrange(1, 5))
    c.pop("name", None)
    return c


# ------------------------------------------------------------------------------------------------ spherical harmonics
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Harmonics:
    """Spherical-harmonic transforms of truncation T on the Gaussian grid the engine uses, FP64, for batches of fields:
    spectra [B, m, n], grids [B, latitude, longitude], south to north."""

    def __init__(self, T):
        self.N, self.M = T, T + 1
        self.nlon = 4
        while self.nlon < 3 * T + 1:
            self.nlon *= 2
        self.nlat = self.nlon // 2
        mu, w = np.polynomial.legendre.leggauss(self.nlat)
        N, M = self.N, self.M
        m, n = np.arange(M)[:, None].astype(float), np.arange(N + 2)[None, :].astype(float)
        with np.errstate(invalid="ignore"):
            eps = np.where(n > m, np.sqrt(np.maximum(n * n - m * m, 0) / np.maximum(4 * n * n - 1, 1)), 0.0)
        P = np.zeros((M, N + 2, self.nlat))
        c = np.sqrt(1 - mu * mu)
        P[0, 0] = 1 / math.sqrt(2.0)
        for k in range(1, M):
            P[k, k] = P[k - 1, k - 1] * math.sqrt((2.0 * k + 1) / (2.0 * k)) * c
        for k in range(1, N + 2):  # degree k of every m < k, then of m = k - 1 from its start alone
            mm = np.arange(min(k, M))
            prev = P[mm, k - 2] if k >= 2 else 0.0
            P[mm, k] = (mu * P[mm, k - 1] - eps[mm, k - 1][:, None] * prev) / eps[mm, k][:, None]
        H = np.zeros((M, M, self.nlat))  # (1 - mu^2) dP/dmu
        H[:] = -n[:, :M, None] * eps[:, 1:, None] * P[:, 1:]
        H[:, 1:] += (n[:, 1:M, None] + 1) * eps[:, 1:M, None] * P[:, : N]
        H *= (n[:, :M] >= m)[:, :, None]
        dev = _device()
        t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(dev)  # noqa: E731
        self.mu, self.w, self.P, self.H = t(mu), t(w), t(P[:, :M]), t(H)
        self.cos = torch.sqrt(1 - self.mu ** 2)
        nn = n[0, :M]
        self.n = t(nn)
        self.im = 1j * t(m)  # [m, 1]
        self.kfac = t(np.where(nn > 0, -A * A / np.maximum(nn * (nn + 1), 1), 0.0))
        self.lapl = t(nn * (nn + 1) / (A * A))
        self.live = t((n[:, :M] >= m).astype(float))

    def _sum(self, c, table):  # [B, m, k] x [m, k, l] -> [B, m, l], complex times real
        B = c.shape[0]
        x = torch.cat([c.real, c.imag]).transpose(0, 1)
        y = torch.matmul(x, table).transpose(0, 1)
        return torch.complex(y[:B].contiguous(), y[B:].contiguous())

    def to_grid(self, four):  # [B, m, lat] -> [B, lat, lon]
        return torch.fft.irfft(four.transpose(1, 2), n=self.nlon, norm="forward")

    def synth(self, spec):
        return self.to_grid(self._sum(spec, self.P))

    def winds(self, z, d):  # u cos(lat), v cos(lat)
        psi, chi = z * self.kfac, d * self.kfac
        U = (self.im * self._sum(chi, self.P) - self._sum(psi, self.H)) / A
        V = (self.im * self._sum(psi, self.P) + self._sum(chi, self.H)) / A
        return self.to_grid(U), self.to_grid(V)

    def fourier(self, grid, weight):
        F = torch.fft.rfft(grid, norm="forward")[..., : self.M] * weight[:, None]
        return F.transpose(1, 2).contiguous()

    def analyse(self, grid):
        return self._sum(self.fourier(grid, self.w), self.P.transpose(1, 2)) * self.live

    def diverge(self, a, b):
        wd = self.w / (1 - self.mu ** 2) / A
        return (self.im * self._sum(self.fourier(a, wd), self.P.transpose(1, 2)) - self._sum(self.fourier(b, wd), self.H.transpose(1, 2))) * self.live


@lru_cache(maxsize=2)
def _harmonics(T):
    return _Harmonics(T)


def _turbulence(T, B, seed, heights, omegas):
    """Balanced turbulence of B members with a divergent part (the gravity waves of a model state): zeta, delta, phi as
    [B, m, n] complex128."""
    h = _harmonics(T)
    g = torch.Generator().manual_seed(int(seed) * 1000003 + T)
    force = max(4, T // 2)

    def noise():
        c = torch.complex(*(torch.randn(B, h.M, h.M, generator=g, dtype=torch.float64) for _ in range(2))).to(h.P.device)
        c[:, 0] = c[:, 0].real.to(c.dtype)
        n = h.n.clamp(min=1)
        shape = torch.sqrt(n ** -3 * n * (n + 1) / (2 * n + 1)) * (h.n >= 1) * (h.n <= force)
        return c * shape * h.live

    z = noise()
    u, v = h.winds(z, 0 * z)
    speed = (torch.hypot(u, v) / h.cos[:, None]).amax(dim=(1, 2), keepdim=True)
    z = z * (30.0 / speed)
    d = 0.2 * 30.0 / speed * noise()
    f = 2 * torch.as_tensor(omegas, dtype=torch.float64, device=h.P.device)[:, None, None] * h.mu[:, None]
    p = h.analyse(f * h.synth(z * h.kfac))
    p[:, 0, 0] = G * math.sqrt(2.0) * torch.as_tensor(heights, dtype=torch.float64, device=h.P.device)
    return z, d, p


def _hill(h, height=500.0):
    """A round mountain at 30 N, 90 E (the height of the surface on the grid)."""
    lat, lon = torch.asin(h.mu)[:, None], 2 * math.pi * torch.arange(h.nlon, dtype=torch.float64, device=h.P.device)[None, :] / h.nlon
    r = torch.sqrt((lat - math.pi / 6) ** 2 + (lon - math.pi / 2) ** 2).clamp(max=math.pi / 9)
    return height * (1 - r * 9 / math.pi)


def _coriolis(h, omegas, tilt):
    lon = 2 * math.pi * torch.arange(h.nlon, dtype=torch.float64, device=h.P.device)[None, :] / h.nlon
    axis = -torch.cos(lon) * h.cos[:, None] * math.sin(tilt) + h.mu[:, None] * math.cos(tilt)
    return 2 * torch.as_tensor(omegas, dtype=torch.float64, device=h.P.device)[:, None, None] * axis


def _nu4(T):
    return A ** 4 / (86400.0 * (T * (T + 1.0)) ** 2)  # e-folding in a day at n = T


def _tendency(h, y, f, hs):
    z, d, p = y[:3]
    U, V = h.winds(z, d)
    Z, F = h.synth(z) + f, h.synth(p)
    a, b = U * Z, V * Z
    E = F + G * hs + (U * U + V * V) / (2 * (1 - h.mu ** 2))[:, None]
    out = [-h.diverge(a, b), h.diverge(b, -a) + h.lapl * h.analyse(E), -h.diverge(U * F, V * F)]
    for k in out:
        k[:, 0, 0] = 0
    if len(y) > 3:
        q = h.synth(y[3])
        out.append(h.analyse(q * h.synth(d)) - h.diverge(U * q, V * q))
    return out


def _integrate(h, y, f, hs, dt, steps, nu4):
    k4 = lambda ev: torch.exp(-nu4 * (ev / A ** 2) ** 2 * dt)  # noqa: E731
    l = h.n * (h.n + 1)
    filt = [k4(l - 2), k4(l - 2), k4(l), k4(l)]
    for x in filt:
        x[0] = 1.0
    for _ in range(steps):
        k1 = _tendency(h, y, f, hs)
        k2 = _tendency(h, [x + 0.5 * dt * k for x, k in zip(y, k1)], f, hs)
        k3 = _tendency(h, [x + 0.5 * dt * k for x, k in zip(y, k2)], f, hs)
        k4_ = _tendency(h, [x + dt * k for x, k in zip(y, k3)], f, hs)
        y = [(x + dt / 6 * (a + 2 * b + 2 * c + e)) * w for x, a, b, c, e, w in zip(y, k1, k2, k3, k4_, filt)]
    return y


# ------------------------------------------------------------------------------------------------ spheres
def _sphere_dt(c):
    return 37800.0 / c["truncation"]  # 900 s at T42, 1800 s at T21


def _sphere_inputs(c, seed):
    B, T = c["members"], c["truncation"]
    h = _harmonics(T)
    y = list(_turbulence(T, B, seed, [8000.0] * B, [OMEGA] * B))
    if c["tracer"]:  # a smooth positive tracer: a background and large-scale waves
        q = _turbulence(T, B, seed + 7, [0.0] * B, [OMEGA] * B)[0]
        q = q / q.abs().amax(dim=(1, 2), keepdim=True) * 0.05
        q[:, 0, 0] = math.sqrt(2.0)
        y.append(q)
    return h, y


class _Sphere:
    def __init__(self, c, seed):
        T, B = c["truncation"], c["members"]
        h, y = _sphere_inputs(c, seed)
        self.case, self.dt = c, _sphere_dt(c)
        self.engine = lw.Sphere(T, diffusion=_nu4(T), members=B, **PRECISION[c["precision"]])
        for b in range(B):
            if c["tilt"]:
                self.engine.set_axis_tilt(c["tilt"], member=b)
            if c["mountain"]:
                self.engine.set_orography_grid(_hill(h).cpu().numpy(), member=b)
        self.state = [x.reshape(B, -1).cpu().numpy()[:, :] for x in y[:3]]
        self.tracer = h.synth(y[3]).cpu().numpy() if c["tracer"] else None

    def run(self):
        s, c = self.engine, self.case
        for b in range(c["members"]):
            s.set_state(self.state[0][b], self.state[1][b], self.state[2][b], member=b)
            if self.tracer is not None:
                s.set_tracer_grid(self.tracer[b], member=b)
        if c["steps"] == 1:
            s.step(self.dt)
        else:
            s.run(c["steps"] * self.dt, self.dt)
        out = [s.get_state(member=b) for b in range(c["members"])]
        if self.tracer is not None:
            out = [(*o, s.tracer_state(member=b)) for b, o in enumerate(out)]
        return [np.stack(x) for x in zip(*out)]


def _sphere_exact(c, seed):
    h, y = _sphere_inputs(c, seed)
    B = c["members"]
    f = _coriolis(h, [OMEGA] * B, c["tilt"])
    hs = _hill(h) if c["mountain"] else 0.0
    y = _integrate(h, y, f, hs, _sphere_dt(c), c["steps"], _nu4(c["truncation"]))
    return [x.reshape(B, -1).cpu().numpy() for x in y]


def _sphere_work(T, members, steps, tracer=False):
    """Per RK4 stage and member: four Legendre syntheses (U, V, vorticity, height) and five analyses at half of the
    latitudes, real FFTs of nine grids; the state (ζ, δ, Φ) in and out once per pass."""
    nlon = 4
    while nlon < 3 * T + 1:
        nlon *= 2
    nlat, tri = nlon // 2, (T + 1) * (T + 2) // 2
    extra = 3 if tracer else 0  # q and δ in, U q, V q, q δ out (the flow's winds are there): 2 + 3 sums
    flops = 4 * ((18 + (10 if tracer else 0)) * nlat * tri + (9 + extra + (2 if tracer else 0)) * nlat * 2.5 * nlon * math.log2(nlon))
    return {"flops": members * steps * flops, "bytes": 2.0 * members * (4 if tracer else 3) * (T + 1) ** 2 * 16}


# ------------------------------------------------------------------------------------------------ ensembles
def _members(c, seed):
    g = np.random.default_rng(seed)
    tr = [21] * c["t21"] + [42] * c["t42"] + [85] * c["t85"]
    return tr, g.uniform(5000.0, 10000.0, len(tr)), [OMEGA * (0.5, 1.0, 2.0)[i % 3] for i in range(len(tr))]


def _ensemble_inputs(c, seed):
    tr, heights, omegas = _members(c, seed)
    at, out = 0, []
    for T, key in ((21, "t21"), (42, "t42"), (85, "t85")):
        n = c[key]
        out.append((T, _turbulence(T, n, seed, heights[at:at + n], omegas[at:at + n]), omegas[at:at + n]))
        at += n
    return tr, heights, omegas, out


def _flat(groups):
    return [np.concatenate([y[f].reshape(-1).cpu().numpy() for y in groups]) for f in range(3)]


def _pinned(n):
    x = torch.empty(2 * n, dtype=torch.float64)
    return (x.pin_memory() if torch.cuda.is_available() else x).numpy().view(np.complex128)


class _Ensemble:
    def __init__(self, c, seed):
        tr, heights, omegas, groups = _ensemble_inputs(c, seed)
        self.engine = lw.Ensemble(tr, [int(seed) * 100000 + i for i in range(len(tr))], heights, omegas, **PRECISION[c["precision"]])
        self.seconds = c["hours"] * 3600.0
        self.state = [_pinned(x.size) for x in _flat([g[1] for g in groups])]
        for a, b in zip(self.state, _flat([g[1] for g in groups])):
            a[:] = b
        self.result = [_pinned(x.size) for x in self.state]

    def run(self):
        self.engine.set_states(*self.state)
        self.engine.run(self.seconds)
        return list(self.engine.get_states(out=self.result))


def _ensemble_exact(c, seed):
    seconds, out = c["hours"] * 3600.0, []
    for T, y, omegas in _ensemble_inputs(c, seed)[3]:
        h = _harmonics(T)
        # the engine's automatic step: the smallest stable step of the group's members
        U, V = h.winds(y[0], y[1])
        wind = (torch.hypot(U, V) / h.cos[:, None]).amax(dim=(1, 2)).cpu().numpy()
        depth = (h.synth(y[2]) / G).amax(dim=(1, 2)).cpu().numpy()
        dt = (1.5 / (T / A * (np.sqrt(G * depth) + wind) + 2 * np.asarray(omegas))).min()
        n = max(1, math.ceil(seconds / dt - 1e-9))
        out.append(_integrate(h, list(y), _coriolis(h, omegas, 0.0), 0.0, seconds / n, n, _nu4(T)))
    return _flat(out)


# ------------------------------------------------------------------------------------------------ planes
class _PlaneSetup:
    """A zonal jet in a mid-latitude channel with seeded height noise and a weak meridional wind."""

    def __init__(self, c, seed):
        nx, ny = c["nx"], c["ny"]
        self.dx = 10000.0 * math.sqrt(1024 * 512 / (nx * ny)) if nx * ny < 1024 * 512 else 10000.0
        self.lx, self.ly = nx * self.dx, ny * self.dx
        self.par = dict(gravity=9.81, depth=1000.0, f0=1e-4, beta=1.6e-11 if self.ly < 6e6 else 1.6e-12, viscosity=c["viscosity"],
                        drag=c["drag"], linear=c["linear"])
        g = np.random.default_rng(seed)
        y = (np.arange(ny) + 0.5) * self.dx
        jet = 15.0 / np.cosh((y - 0.5 * self.ly) / (0.12 * self.ly)) ** 2
        f = self.par["f0"] + self.par["beta"] * (y - 0.5 * self.ly)
        slope = np.cumsum(-f * jet * self.dx / 9.81)
        self.h = 1000.0 + (slope - slope.mean())[:, None] + 0.5 * g.standard_normal((ny, nx))
        self.u = jet[:, None] + 0.1 * g.standard_normal((ny, nx))
        self.v = 0.1 * g.standard_normal((ny + 1, nx))
        self.v[0] = self.v[ny] = 0.0
        self.dt = 0.25 * self.dx / (math.sqrt(9.81 * self.h.max()) + 20.0)
        self.seconds = c["steps"] * self.dt


class _Plane:
    def __init__(self, c, seed):
        p = self.setup = _PlaneSetup(c, seed)
        self.engine = lw.Plane(c["nx"], c["ny"], p.lx, p.ly, **p.par)

    def run(self):
        e, p = self.engine, self.setup
        e.set_h_from_grid(p.h).set_u_from_grid(p.u).set_v_from_grid(p.v)
        e.run(p.seconds, p.dt)
        return list(e.get())


def _plane_tendency(p, nx, ny, h, u, v):
    """C-grid shallow water, periodic in x with walls at both y ends: h at centres, u at west faces, v at south faces."""
    dx, dy = p.lx / nx, p.ly / ny
    a, linear = p.par, p.par["linear"]
    west, east = (lambda x: torch.roll(x, 1, 1)), (lambda x: torch.roll(x, -1, 1))
    j = torch.arange(ny + 1, dtype=torch.float64, device=h.device)[:, None]
    eta = a["f0"] + a["beta"] * (j * dy - 0.5 * p.ly) + torch.zeros_like(v)
    bern = a["gravity"] * h
    if not linear:
        eta = eta + (v - west(v)) / dx
        eta[1:ny] -= (u[1:] - u[:-1]) / dy
        bern = bern + 0.5 * (0.5 * (u * u + east(u) ** 2) + 0.5 * (v[:-1] ** 2 + v[1:] ** 2))
    vbar = 0.25 * (west(v[:-1]) + v[:-1] + west(v[1:]) + v[1:])
    du = 0.5 * (eta[:-1] + eta[1:]) * vbar - (bern - west(bern)) / dx - a["drag"] * u
    dv = torch.zeros_like(v)
    ubar = 0.25 * (u[:-1] + east(u[:-1]) + u[1:] + east(u[1:]))
    e = eta[1:ny]
    dv[1:ny] = -0.5 * (e + east(e)) * ubar - (bern[1:] - bern[:-1]) / dy - a["drag"] * v[1:ny]
    if a["viscosity"]:
        up, um = torch.cat([u[1:], u[-1:]]), torch.cat([u[:1], u[:-1]])
        du = du + a["viscosity"] * ((east(u) - 2 * u + west(u)) / dx ** 2 + (up - 2 * u + um) / dy ** 2)
        w = v[1:ny]
        dv[1:ny] += a["viscosity"] * ((east(w) - 2 * w + west(w)) / dx ** 2 + (v[2:] - 2 * w + v[:-2]) / dy ** 2)
    hx = a["depth"] if linear else 0.5 * (west(h) + h)
    fx = hx * u
    fy = torch.zeros_like(v)
    fy[1:ny] = (a["depth"] if linear else 0.5 * (h[1:] + h[:-1])) * v[1:ny]
    return -((east(fx) - fx) / dx + (fy[1:] - fy[:-1]) / dy), du, dv


def _plane_exact(c, seed):
    p = _PlaneSetup(c, seed)
    y = [torch.from_numpy(x).to(_device()) for x in (p.h, p.u, p.v)]
    n = max(1, math.ceil(p.seconds / p.dt - 1e-9))
    dt = p.seconds / n
    for _ in range(n):
        k1 = _plane_tendency(p, c["nx"], c["ny"], *y)
        k2 = _plane_tendency(p, c["nx"], c["ny"], *(x + 0.5 * dt * k for x, k in zip(y, k1)))
        k3 = _plane_tendency(p, c["nx"], c["ny"], *(x + 0.5 * dt * k for x, k in zip(y, k2)))
        k4 = _plane_tendency(p, c["nx"], c["ny"], *(x + dt * k for x, k in zip(y, k3)))
        y = [x + dt / 6 * (a + 2 * b + 2 * d + e) for x, a, b, d, e in zip(y, k1, k2, k3, k4)]
    return [x.cpu().numpy() for x in y]


# ------------------------------------------------------------------------------------------------ networks
def _network(c, seed):
    """Weights as the surrogate starts with them (normal, 1/sqrt(fan in)), normalised states and increments."""
    g = torch.Generator(device=_device()).manual_seed(int(seed))
    f, h = c["features"], c["hidden"]
    shapes = [(h, f), (h, h), (h, h), (f, h)]
    r = lambda *s: torch.randn(*s, generator=g, device=_device())  # noqa: E731
    W = [r(*s) / math.sqrt(s[1]) for s in shapes]
    b = [0.1 * r(s[0]) for s in shapes]
    return W, b, r(c["batch"], f), r(c["batch"], f)


class _Network:
    def __init__(self, c, seed):
        W, b, x, t = _network(c, seed)
        self.train = c["kind"] == "train"
        self.net = lw.Mlp(c["features"], c["hidden"], c["features"], max_batch=c["batch"], seed=1)
        for k in range(4):
            self.net.set_layer(k, W[k].cpu().numpy(), b[k].cpu().numpy())
        self.x, self.t = x.cpu().numpy(), t.cpu().numpy()

    def run(self):
        if not self.train:
            return self.net.forward(self.x)
        loss = self.net.backward(self.x, self.t)
        grads = [self.net.grad(k) for k in range(4)]
        self.net.adam(lr=3e-4)
        return {"loss": loss, "grads": grads, "weights": [self.net.get_layer(k) for k in range(4)]}


def _network_exact(c, seed):
    W, b, x, t = ([y.double() for y in v] if isinstance(v, list) else v.double() for v in _network(c, seed))
    cdf = lambda z: 0.5 * (1 + torch.erf(z / math.sqrt(2.0)))  # noqa: E731
    act, zs = [x], []
    for k in range(3):
        zs.append(act[-1] @ W[k].T + b[k])
        act.append(zs[-1] * cdf(zs[-1]))
    y = act[-1] @ W[3].T + b[3]
    if c["kind"] == "forward":
        return y.cpu().numpy()
    loss = float(0.5 * ((y - t) ** 2).sum() / c["batch"])
    d, grads = (y - t) / c["batch"], []
    for k in range(3, -1, -1):
        grads.insert(0, (d.T @ act[k], d.sum(0)))
        if k:
            z = zs[k - 1]
            d = (d @ W[k]) * (cdf(z) + z * torch.exp(-0.5 * z * z) / math.sqrt(2 * math.pi))
    step = lambda w, g: (w - 3e-4 * g / (g.abs() + 1e-8)).cpu().numpy()  # noqa: E731  (Adam's first step)
    return {"loss": loss, "grads": [tuple(v.cpu().numpy() for v in g) for g in grads],
            "weights": [(step(W[k], grads[k][0]), step(b[k], grads[k][1])) for k in range(4)]}


# ------------------------------------------------------------------------------------------------ the interface
def prepare(case, seed):
    kind = case["kind"]
    return {"sphere": _Sphere, "ensemble": _Ensemble, "plane": _Plane, "forward": _Network, "train": _Network}[kind](case, seed)


def run(state):
    return state.run()


def work(case):
    kind = case["kind"]
    if kind == "sphere":
        return _sphere_work(case["truncation"], case["members"], case["steps"], case["tracer"])
    if kind == "ensemble":
        total = {"flops": 0.0, "bytes": 0.0}
        for T, key in ((21, "t21"), (42, "t42"), (85, "t85")):
            # the automatic step of the shallowest to deepest members, at the fastest rotation
            steps = math.ceil(case["hours"] * 3600.0 * (T / A * (math.sqrt(G * 10000.0) + 45.0) + 4 * OMEGA) / 1.5)
            w = _sphere_work(T, case[key], steps)
            total = {k: total[k] + w[k] for k in total}
        return total
    if kind == "plane":
        cells = case["nx"] * case["ny"]
        return {"flops": 4.0 * case["steps"] * cells * (58 + (16 if case["viscosity"] else 0)), "bytes": 48.0 * cells}
    f, h, b = case["features"], case["hidden"], case["batch"]
    weights = 2 * f * h + 2 * h * h
    if kind == "forward":
        return {"flops": 2.0 * b * weights, "bytes": 8.0 * b * f + 2.0 * weights}
    return {"flops": 2.0 * b * (3 * weights - f * h), "bytes": 8.0 * b * f + 28.0 * weights}


def exact(case, seed):
    kind = case["kind"]
    return {"sphere": _sphere_exact, "ensemble": _ensemble_exact, "plane": _plane_exact, "forward": _network_exact,
            "train": _network_exact}[kind](case, seed)
