"""What the framework is timed on: model runs through its public entry points
(qgw_gb300.capi), from one step of a 64 x 64 basin to steps of a 2048 x 2048
one, in both precisions.

A case is a dict:
  kind   "steps": a run from an initial state to its next output -- set q (on
         the device) and the clock, n steps, psi and q out;
         "host": timestep(q) on the caller's own host array, n steps a call;
         "invert": a stored q in, its psi and energy budget out;
         "ensemble": members of uneven sizes advanced together
  prec   0: FP64, 1: compensated FP32 (its fields go on in single precision,
         as vars.nc stores them)
  NX, NY, nl, n
  bc     wall rule bc_fac (0 free slip, 1 no slip), -1: doubly periodic
  hyper  1: biharmonic-type chain on psi (n_hyper = 4), 0: viscosity on q
  topo   1: the analytic shelf;  ring: radius of the stochastic forcing (0: none)
  ic     "noise": white q (std 1e-7 1/s); "eddies": basin and mesoscale waves,
         weaker in each layer down, with that noise on top
"""
import math
import random

import numpy as np
import torch

LX, F0, BETA, TAU0, DRAG = 4.0e6, 1e-4, 2e-11, 8e-5, 1e-7


def case(name, kind, prec, NX, NY, nl, n, bc=0.0, hyper=1, topo=0, ring=0, ic="eddies", dt=600.0, mseed=0):
    c = dict(kind=kind, prec=prec, NX=NX, NY=NY, nl=nl, n=n, bc=bc, hyper=hyper, topo=topo, ring=ring, ic=ic, dt=dt,
             mseed=mseed)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a host model that owns q steps a 64^2 test basin
        case("host_fp64_64x3", "host", 0, 64, 64, 3, 1, hyper=0, dt=1200.0),
        # a day of the 3-layer double gyre, then output: the everyday research run
        case("gyre_fp64_256x3", "steps", 0, 256, 256, 3, 72, hyper=0, dt=1200.0, ic="noise"),
        # the eddy-resolving 10-layer basin in plain FP64, the headline run
        case("basin_fp64_1024x10", "steps", 0, 1024, 1024, 10, 10, ic="noise"),
        # the same as the time step of a host program that keeps q itself
        case("host_fp64_1024x10", "host", 0, 1024, 1024, 10, 1),
        # the largest grid
        case("basin_fp64_2048x6", "steps", 0, 2048, 2048, 6, 4, dt=300.0),
        # not square, not powers of two; no-slip walls over a shelf
        case("shelf_fp64_384x240x3", "steps", 0, 384, 240, 3, 20, bc=1.0, hyper=0, topo=1),
        # doubly periodic turbulence
        case("periodic_fp64_512x5", "steps", 0, 512, 512, 5, 10, bc=-1.0),
        # odd sizes: grids taken from a regional domain as it comes
        case("odd_fp64_301x207x4", "steps", 0, 301, 207, 4, 10),
        # many layers on a small grid, compensated FP32
        case("basin_fp32c_256x16", "steps", 1, 256, 256, 16, 50),
        # the headline run, compensated FP32
        case("basin_fp32c_1024x10", "steps", 1, 1024, 1024, 10, 40, ic="noise"),
        # a parameter study: 16 uneven basins at once
        case("ensemble_fp32c_16", "ensemble", 1, 0, 0, 0, 10, mseed=4),
        # diagnostics of a stored state: PV inversion and energy budget
        case("invert_fp64_768x8", "invert", 0, 768, 768, 8, 1),
    ]


def smooth_even(n):
    """The even number at or below n with n/2 a product of 2, 3, 5 and 7."""
    while True:
        n -= n % 2
        h = n // 2
        for f in (2, 3, 5, 7):
            while h % f == 0:
                h //= f
        if h == 1:
            return n
        n -= 2


def draw(rng):
    kind = rng.choice(["steps"] * 6 + ["host"] * 2 + ["invert", "ensemble"])
    if kind == "ensemble":
        return case("", kind, 1, 0, 0, 0, rng.randint(4, 20), mseed=rng.randrange(1000, 10**6))
    prec = rng.choice([0, 0, 1])
    NX = int(round(math.exp(rng.uniform(math.log(40), math.log(1400)))))
    NY = max(40, min(1400, int(round(NX * math.exp(rng.uniform(-0.7, 0.7))))))
    bc = rng.choice([0.0, 0.0, 0.0, 1.0, 0.5, -1.0])
    form = rng.choice(["smooth", "smooth", "pow2", "any"])
    if bc == -1.0 or form == "smooth":
        NX, NY = smooth_even(NX), smooth_even(NY)
    elif form == "pow2":
        NX, NY = (1 << int(round(math.log2(v))) for v in (NX, NY))
    if bc == -1.0:
        NY = NX
    nl = max(1, min(20, int(round(math.exp(rng.uniform(0, math.log(20)))))))
    nl = max(1, min(nl, 10_000_000 // (NX * NY)))
    weight = 6 if smooth_even(NX) != NX or smooth_even(NY) != NY else 1
    n = 1 if kind != "steps" else max(1, min(rng.randint(5, 60), 80_000_000 // (NX * NY * nl * weight)))
    ring = rng.randint(4, 12) if bc == -1.0 and rng.random() < 0.4 else 0
    hyper = rng.choice([0, 1])
    topo = 1 if bc >= 0 and rng.random() < 0.25 else 0
    dt = 1200.0 if NX <= 256 else 600.0 if NX <= 1024 else 300.0
    return case("", kind, prec, NX, NY, nl, n, bc, hyper, topo, ring, rng.choice(["noise", "eddies"]), dt)


def layers(nl):
    """Thicknesses (stretched, 4000 m in all) and N2 of the interfaces."""
    if nl == 1:
        return [4000.0], [1.0]
    if nl == 3:
        dh, gp = [500.0, 1000.0, 2500.0], [0.02, 0.01]
    else:
        r = 1.3
        d0 = 4000.0 * (r - 1.0) / (r ** nl - 1.0)
        dh = [d0 * r ** k for k in range(nl)]
        gp = [0.02 * 0.1 ** (l / max(1, nl - 2)) for l in range(nl - 1)]
    return dh, [gp[l] / (0.5 * (dh[l] + dh[l + 1])) for l in range(nl - 1)]


def params(c):
    dh, N2 = layers(c["nl"])
    p = dict(NX=c["NX"], NY=c["NY"], nl=c["nl"], Lx=LX, dh=dh, N2=N2, f0=F0, beta=BETA, tau0=TAU0, forc_mode=2.0,
             nu=0.0 if c["hyper"] else 50.0, n_hyper=4 if c["hyper"] else 0, nu_hyper=1e9 if c["hyper"] else 0.0,
             hEkb=2.0 * DRAG * dh[-1] / F0, bc_fac=c["bc"], cfl=0.2, tend=1e12, dt_out=1e12, dt=c["dt"])
    if c["topo"]:
        p.update(h_topo=300.0, w_topo=4e5)
    if c["ring"]:
        p.update(k_f=2 * math.pi * c["ring"] / LX, sigma_f=1e-12)
    return p


def members(c):
    """The uneven members of an ensemble case, each a steps case."""
    r = random.Random(c["mseed"])
    return [case("", "steps", 1, N, N, r.choice([2, 3, 5, 10]), c["n"], ic=r.choice(["noise", "eddies"]))
            for N in (r.choice([64, 96, 128, 192, 256, 384, 512]) for _ in range(16))]


def interior(c):
    d = 0 if c["bc"] == -1.0 else 1
    return c["nl"], c["NY"] - d, c["NX"] - d


def device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def initial(c, seed):
    """q of the interior points with a zero ring around it, on the GPU."""
    nl, ny, nx = interior(c)
    dev = device()
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    rnd = dict(generator=g, device=dev, dtype=torch.float64)
    q = torch.zeros(nl, ny + 2, nx + 2, device=dev, dtype=torch.float64)
    q[:, 1:-1, 1:-1] = 1e-7 * torch.randn(nl, ny, nx, **rnd)
    if c["ic"] == "eddies":
        x = torch.arange(nx, device=dev, dtype=torch.float64) * (2 * math.pi / nx)
        y = torch.arange(ny, device=dev, dtype=torch.float64) * (2 * math.pi / ny)
        for _ in range(8):
            u = torch.rand(5, **rnd).tolist()
            k, l = 1 + int(12 * u[0]), 1 + int(12 * u[1])
            wave = torch.outer(torch.sin(l * y + 6.28 * u[2]), torch.sin(k * x + 6.28 * u[3]))
            amp = 2e-6 * u[4] * 0.6 ** torch.arange(nl, device=dev, dtype=torch.float64)
            q[:, 1:-1, 1:-1] += amp[:, None, None] * wave
    return q


def host_array(shape):
    t = torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return t.numpy()


def prepare(c, seed):
    from qgw_gb300 import capi
    s = {"case": c}
    if c["kind"] == "ensemble":
        ms = members(c)
        s["ens"] = capi.Ensemble([params(m) for m in ms], capi.FP32C)
        s["q0"] = [initial(m, seed * 64 + i).cpu().numpy() for i, m in enumerate(ms)]
        s["dt"] = [m["dt"] for m in ms]
        return s
    r = s["run"] = capi.Run(params(c), capi.FP32C if c["prec"] else capi.FP64)
    q = initial(c, seed)
    s["psi"], s["q"] = host_array(r.shape), host_array(r.shape)
    if c["prec"]:
        s["out"] = [torch.empty(r.shape, dtype=torch.float32) for _ in range(2)]
    if c["kind"] == "steps":
        s["q0"] = q
    else:
        s["q0"] = host_array(r.shape)
        s["q0"][:] = q.cpu().numpy()
        r.set_q(s["q0"])
        r.fix_dt(c["dt"])
    torch.cuda.synchronize()
    return s


def single(s, *fields):
    """Fields as vars.nc stores them."""
    return [o.copy_(torch.from_numpy(f)) for o, f in zip(s["out"], fields)]


def run(s):
    c = s["case"]
    if c["kind"] == "ensemble":
        e = s["ens"]
        for i in range(len(e)):
            e.set_q(i, s["q0"][i])
            e.fix_dt(i, s["dt"][i])
        e.step(c["n"])
        return [[torch.from_numpy(f).float() for f in e.get(i)] for i in range(len(e))]
    r = s["run"]
    if c["ring"]:
        r.set_forcing_seed(1)
    if c["kind"] == "host":
        r.step_host(c["n"], s["q0"], s["q"])
        return single(s, s["q"]) if c["prec"] else [s["q"]]
    if c["kind"] == "invert":
        r.set_q(s["q0"])
        r.get(s["psi"], s["q"])
        b = r.budget()
        fields = single(s, s["psi"], s["q"]) if c["prec"] else [s["psi"], s["q"]]
        budget = np.array([b[k] for k in ("ke", "energy", "enstrophy", "wind_work")])
        return fields + [budget.astype(np.float32) if c["prec"] else budget]
    r.set_q_device(s["q0"].data_ptr())
    r.fix_dt(c["dt"])
    r.step(c["n"])
    r.get(s["psi"], s["q"])
    return single(s, s["psi"], s["q"]) if c["prec"] else [s["psi"], s["q"]]


def work(c):
    """q in, psi and q out once a call; in each step q and the two older
    tendencies are read, q and the new one written, psi made and used, all in
    the run's own precision, by four 1-D transforms, the layer sums and the
    stencils."""
    if c["kind"] == "ensemble":
        ws = [work(m) for m in members(c)]
        return {k: sum(w[k] for w in ws) for k in ws[0]}
    nl, ny, nx = interior(c)
    pts = nl * ny * nx
    elem = 4 if c["prec"] else 8
    steps = 0 if c["kind"] == "invert" else c["n"]
    transforms = 5.0 * (math.log2(nx + 1) + math.log2(ny + 1)) + 4.0 * nl
    passes = max(1, steps)
    edge = 16 if c["kind"] == "host" else 24
    return {"bytes": pts * (edge + steps * 7.0 * elem), "flops": pts * (passes * transforms + steps * 70.0)}


# ------------------------------------------------------------------- exact
def vertical_modes(p):
    nl = p["nl"]
    if nl == 1:
        one = np.ones((1, 1))
        return one, one, np.zeros(1)
    dh = np.array(p["dh"])
    G = np.zeros((nl, nl))
    for l in range(nl - 1):
        s = F0 * F0 / p["N2"][l] / (0.5 * (dh[l] + dh[l + 1]))
        G[l, l + 1] -= s / dh[l]
        G[l, l] += s / dh[l]
        G[l + 1, l] -= s / dh[l + 1]
        G[l + 1, l + 1] += s / dh[l + 1]
    sd = np.sqrt(dh)
    sym = sd[:, None] * G / sd[None, :]
    w, u = np.linalg.eigh(0.5 * (sym + sym.T))
    vr = u / sd[:, None]
    vr *= np.where(vr[0] > 0, 1.0, -1.0) * np.sqrt(dh.sum() / (dh[:, None] * vr * vr).sum(0))
    vl = vr * dh[:, None]
    vl /= (vl * vr).sum(0)
    w[0] = 0.0
    return vl.T.copy(), vr, w  # layers -> modes, modes -> layers, 1/Rd^2


class Model:
    """The reference's step in torch, 64 bits, fields without their ring."""

    def __init__(self, c, p):
        self.c, self.p, self.dev = c, p, device()
        self.nl, self.ny, self.nx = interior(c)
        self.per = c["bc"] == -1.0
        self.D = LX / c["NX"]
        self.Ly = c["NY"] * self.D
        self.l2m, self.m2l, ird = (self.t(v) for v in vertical_modes(p))
        if self.per:
            kx = 2 * math.pi / LX * torch.arange(self.nx // 2 + 1, dtype=torch.float64, device=self.dev)
            ky = 2 * math.pi / LX * torch.fft.fftfreq(self.ny, 1.0 / self.ny, dtype=torch.float64, device=self.dev)
        else:
            kx = math.pi / LX * torch.arange(1, self.nx + 1, dtype=torch.float64, device=self.dev)
            ky = math.pi / LX * torch.arange(1, self.ny + 1, dtype=torch.float64, device=self.dev)
        self.fact = -((kx ** 2)[None, None, :] + (ky ** 2)[None, :, None] + ird[:, None, None])
        off = -1 if self.per else 0
        self.X = (np.arange(self.nx + 2) + off) * self.D
        self.Y = (np.arange(self.ny + 2) + off) * self.D
        mode = p["forc_mode"] * math.pi
        self.wind = self.t(-TAU0 / p["dh"][0] * mode / self.Ly * np.sin(mode * self.Y[1:-1] / self.Ly))[:, None]
        self.topo = None
        if c["topo"]:
            sh = lambda x: 1 - np.exp(-(x * x) / (2 * p["w_topo"] ** 2))  # noqa: E731
            inside = (sh(self.Y) * sh(self.Ly - self.Y))[:, None] * (sh(self.X) * sh(LX - self.X))[None, :]
            self.topo = self.t(p["h_topo"] * (1 - inside))[None]

    def t(self, v):
        return torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float64, device=self.dev)

    def dst(self, v):
        """Sine transform (2 sum x sin) along the last axis."""
        n = v.shape[-1]
        z = torch.zeros(v.shape[:-1] + (1,), dtype=torch.float64, device=self.dev)
        return -torch.fft.rfft(torch.cat([z, v, z, -v.flip(-1)], -1)).imag[..., 1:n + 1]

    def invert(self, q):
        m = torch.einsum("ml,lyx->myx", self.l2m, q)
        out = torch.empty_like(m)
        for k in range(self.nl):  # a mode at a time: the work arrays of all would not be small
            if self.per:
                f = self.fact[k].clone()
                f[0, 0] = 1.0
                s = torch.fft.rfft2(m[k]) / f
                s[0, 0] = 0
                out[k] = torch.fft.irfft2(s, s=(self.ny, self.nx))
            else:
                s = self.dst(self.dst(m[k]).T.contiguous()).T / self.fact[k]
                s = self.dst(self.dst(s.contiguous()).T.contiguous()).T
                out[k] = s / (4.0 * (self.nx + 1) * (self.ny + 1))
        return torch.einsum("lm,myx->lyx", self.m2l, out)

    def ring(self, f, psi=None):
        """f with its ring: wrapped, or at walls 0 (psi None) or the vorticity of the wall rule."""
        if self.per:
            f = torch.cat([f[:, -1:], f, f[:, :1]], 1)
            return torch.cat([f[:, :, -1:], f, f[:, :, :1]], 2)
        g = torch.nn.functional.pad(f, (1, 1, 1, 1))
        if psi is not None and self.c["bc"] != 0:
            k = 2 * self.c["bc"] / self.D ** 2
            g[:, 0, 1:-1], g[:, -1, 1:-1] = k * psi[:, 0], k * psi[:, -1]
            g[:, 1:-1, 0], g[:, 1:-1, -1] = k * psi[:, :, 0], k * psi[:, :, -1]
        return g

    def lap(self, g):
        return ((g[:, 1:-1, 2:] + g[:, 1:-1, :-2]) + (g[:, 2:, 1:-1] + g[:, :-2, 1:-1])
                - 4 * g[:, 1:-1, 1:-1]) / self.D ** 2

    def jacobian(self, p, q):
        def at(f, dx, dy):
            return f[:, 1 + dy:f.shape[1] - 1 + dy, 1 + dx:f.shape[2] - 1 + dx]
        E, W, N, S = (1, 0), (-1, 0), (0, 1), (0, -1)
        NE, NW, SE, SW = (1, 1), (-1, 1), (1, -1), (-1, -1)
        P, Q = (lambda d: at(p, *d)), (lambda d: at(q, *d))
        return ((P(E) - P(W)) * (Q(N) - Q(S)) + (P(S) - P(N)) * (Q(E) - Q(W))
                + P(E) * (Q(NE) - Q(SE)) - P(W) * (Q(NW) - Q(SW)) - P(N) * (Q(NE) - Q(NW)) + P(S) * (Q(SE) - Q(SW))
                + Q(N) * (P(NE) - P(NW)) - Q(S) * (P(SE) - P(SW)) - Q(E) * (P(NE) - P(SE)) + Q(W) * (P(NW) - P(SW))
                ) / (12.0 * self.D ** 2)

    def rhs(self, q, psi):
        p = self.p
        gp, gq = self.ring(psi), self.ring(q, psi)
        f = -self.jacobian(gp, gq) - BETA * (gp[:, 1:-1, 2:] - gp[:, 1:-1, :-2]) / (2 * self.D)
        if p["nu"]:
            f += p["nu"] * self.lap(gq)
        if p["nu_hyper"]:
            g = gp
            for _ in range(p["n_hyper"] // 2 + 1):
                l = self.lap(g)
                g = self.ring(l, psi)
            f += (-1.0) ** (p["n_hyper"] // 2 - 1) * p["nu_hyper"] * l
        f[0] += self.wind
        f[-1] -= p["hEkb"] * F0 / (2 * p["dh"][-1]) * self.lap(gp[-1:])[0]
        if self.topo is not None:
            f[-1] -= self.jacobian(gp[-1:], self.topo)[0] * (F0 / p["dh"][-1])
        return f

    def steps(self, q, n):
        dt = dt0 = dt1 = DT = self.c["dt"]
        f1 = f2 = torch.zeros_like(q)
        for _ in range(n):
            psi = self.invert(q)
            f0 = self.rhs(q, psi)
            g = self.ring(psi)
            u = max(float((g[:, 1:-1, 2:] - psi).abs().max()), float((g[:, 2:, 1:-1] - psi).abs().max())) / self.D
            dt1, dt0 = dt0, dt
            dt = min(2 * dt, DT, p_cfl(self.p, self.D, u))
            c0 = dt * (2 * dt * dt + 3 * dt * (2 * dt0 + dt1) + 6 * dt0 * (dt0 + dt1)) / (6 * dt0 * (dt0 + dt1))
            c1 = dt * dt * (-dt / 3 - dt0 / 2 - dt1 / 2) / (dt0 * dt1)
            c2 = dt * dt * (dt / 3 + dt0 / 2) / (dt1 * (dt0 + dt1))
            q = q + c0 * f0 + c1 * f1 + c2 * f2
            f1, f2 = f0, f1
        return q

    def budget(self, q, psi):
        w = self.t(np.array(self.p["dh"]) / sum(self.p["dh"]))[:, None, None]
        g = self.ring(psi)
        u, v = (g[:, 1:-1, 2:] - psi) / self.D, (g[:, 2:, 1:-1] - psi) / self.D
        sums = [(w * 0.5 * (u * u + v * v)).sum(), -(w * psi * q).sum(), (w * q * q).sum(),
                -(w[0] * psi[0] * self.wind).sum()]
        return np.array([float(x) for x in sums]) * (self.D ** 2 / (LX * self.Ly))


def p_cfl(p, delta, u):
    return p["cfl"] * delta / u if u else 1e30


def exact(c, seed):
    if c["kind"] == "ensemble":
        return [exact(m, seed * 64 + i) for i, m in enumerate(members(c))]
    if c["ring"]:
        return None  # its noise is the C library's rand()
    m = Model(c, params(c))
    q = initial(c, seed)[:, 1:-1, 1:-1].contiguous()
    if c["kind"] != "invert":
        q = m.steps(q, c["n"])
    psi = m.invert(q)
    full_psi, full_q = m.ring(psi), m.ring(q, psi)
    if c["kind"] == "host":
        return [full_q]
    return [full_psi, full_q] + ([m.budget(q, psi)] if c["kind"] == "invert" else [])
