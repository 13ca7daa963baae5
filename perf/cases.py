"""Timed cases: the work that programs on this engine have it do, through its
public entry points.

A case is a dict of plain values.  ``prepare`` builds what a program holds
before the call (grids set up from decks, with a developed field in them),
``run`` is one pass (time steps, then the read-out of the results), ``exact``
gives the same results from a plain FP64 restatement of the physics in torch,
and ``work`` counts the bytes and operations a pass cannot do without.

Kinds of case:
  scatterer   vacuum with a dielectric sphere, CPML, one point source
  dispersive  Drude-Lorentz spheres in vacuum, CPML, TF/SF Gaussian beam, six
              planar ports with a DFT around the beam box
  laser       disordered photonic crystal in a four-level gain medium, CPML,
              seed dipole, spherical port with a DFT
  ensemble    several laser realizations of uneven size stepped as one batch
  served      a stream of small jobs of all three physics through the server,
              set up from host data, stepped and read out inside the pass
"""
import ctypes
import math

import numpy as np
import torch

import cpsfdtd_b200 as cps
from cpsfdtd_b200 import decks

EPS0, MU0, C0, PI = decks.EPS0, decks.MU0, decks.C0, decks.PI
H_PLANCK = 6.62607004081e-34
EZ, ALL = "Ez", "all"


def _case(kind, nx, ny, nz, npml, dtype, steps, path="fused", nfreq=0, read=ALL, **more):
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, npml=npml, dtype=dtype, steps=steps, path=path, nfreq=nfreq,
                read=read, **more)


def listed():
    c = []

    def add(name, *a, **k):
        c.append(dict(_case(*a, **k), name=name))

    # a quick study on a small grid: every array fits L2, a step is a handful of short launches
    add("scatterer_48_f32", "scatterer", 48, 48, 48, 5, "f32", 200)
    # the FP64 path in the reference's order of routines, on the size of its plain scatterer deck
    add("scatterer_96_f64_plain", "scatterer", 96, 96, 96, 10, "f64", 100, path="plain")
    # passive scattering on a large box with odd, unequal edges
    add("scatterer_301x419x262_f32", "scatterer", 301, 419, 262, 10, "f32", 256, read=EZ)
    # the dispersive-scattering deck at its size
    add("dispersive_256_f32", "dispersive", 256, 256, 256, 12, "f32", 512, nfreq=16, read=EZ)
    # dispersive scattering in FP64, for users who check the FP32 results
    add("dispersive_165x150x181_f64", "dispersive", 165, 150, 181, 9, "f64", 128, nfreq=8)
    # the same physics driven by a main loop that calls one routine per term, with recording on
    add("main_loop_145x118x131_f32", "dispersive", 145, 118, 131, 8, "f32", 128, path="calls", nfreq=8)
    # the photonic-crystal laser at its size: the largest grid
    add("laser_384_f32", "laser", 384, 384, 384, 16, "f32", 256, nfreq=8, read=EZ)
    # a laser cavity of ordinary size with unequal edges
    add("laser_150x117x98_f32", "laser", 150, 117, 98, 8, "f32", 256, nfreq=16)
    # the laser in FP64
    add("laser_176_f64", "laser", 176, 176, 176, 9, "f64", 64, nfreq=8)
    # a Monte-Carlo ensemble of small lasers as one batch
    add("ensemble_16_f32", "ensemble", 64, 128, 16, 8, "f32", 192, nfreq=16, read="ports")
    # jobs of uneven length through the server, from host data to spectra
    add("served_6_f32", "served", 48, 96, 6, 8, "f32", 256, nfreq=8, read="ports")
    return c


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def edges(lo, hi):
        n = log(lo, hi)
        return [max(lo, min(hi, int(n * rng.uniform(0.75, 1.3)))) for _ in range(3)]

    kind = rng.choice(["scatterer", "scatterer", "dispersive", "dispersive", "laser", "laser", "ensemble", "served"])
    if kind == "scatterer":
        f64 = rng.random() < 0.4
        e = edges(36, 160 if f64 else 400)
        cells = e[0] * e[1] * e[2]
        steps = max(24, min(200, int(4e9 / cells))) if f64 else max(64, min(256, int(8e9 / cells)))
        return _case("scatterer", *e, rng.randint(5, 10), "f64" if f64 else "f32", steps,
                     path=rng.choice(["plain", "fused"]) if f64 else "fused", read=ALL if cells < 4e6 else EZ)
    if kind == "dispersive":
        f64 = rng.random() < 0.3
        e = edges(64, 190 if f64 else 256)
        cells = e[0] * e[1] * e[2]
        return _case("dispersive", *e, rng.randint(6, 12), "f64" if f64 else "f32",
                     max(48, min(256, int(3e9 / cells))), path=rng.choice(["fused", "fused", "calls"]),
                     nfreq=rng.choice([5, 8, 16, 33]), read=ALL if cells < 4e6 else EZ)
    if kind == "laser":
        f64 = rng.random() < 0.3
        e = edges(56, 176 if f64 else 320)
        cells = e[0] * e[1] * e[2]
        return _case("laser", *e, rng.randint(6, 12), "f64" if f64 else "f32", max(48, min(256, int(2e9 / cells))),
                     nfreq=rng.choice([4, 8, 16]), read=ALL if cells < 4e6 else EZ)
    if kind == "ensemble":
        lo = rng.randint(48, 64)
        return _case("ensemble", lo, rng.randint(96, 128), rng.randint(6, 20), rng.randint(6, 8), "f32",
                     rng.randint(64, 192), nfreq=rng.choice([4, 8, 16]), read="ports")
    lo = rng.randint(40, 56)
    return _case("served", lo, rng.randint(72, 96), rng.randint(4, 6), rng.randint(5, 8), "f32",
                 rng.randint(128, 256), nfreq=rng.choice([4, 8]), read="ports")


# ------------------------------------------------------------------- decks

def _spheres(deck, centres, radius, mat, background=0):
    deck.ids = decks.rasterize_spheres(deck.shape3, deck.dx, centres, radius, mat, background=background)


def _wave(deck, steps):
    return decks.gaussian_sine(4 * steps + 2, deck.dt, 600e-9, 5e-15, 7e-15)


def _scatterer(nx, ny, nz, npml, steps, seed):
    d = 10e-9
    rng = np.random.Generator(np.random.PCG64(seed))
    dk = decks.Deck(nx, ny, nz, d, d, d, media=[(1.0, 1.0, 0.0, 0.0), (2.25, 1.0, 0.0, 0.0)])
    c = np.array([[nx, ny, nz]]) / 2.0 + rng.uniform(-2, 2, size=(1, 3))
    _spheres(dk, c, 0.2 * min(nx, ny, nz), 1)
    dk.pml = decks.pml_params(npml)
    dk.sources = [(decks.COMP["Ez"], nx // 3, ny // 2, nz // 2, _wave(dk, steps))]
    dk.ports = [decks.Port("plain", dict(dir="z", position=(nz // 2 + 0.5) * d, w1=0.5 * d, w2=(nx - 0.5) * d,
                                         h1=(ny // 2 + 0.5) * d, h2=(ny // 2 + 0.5) * d))]
    return dk


def _dispersive(nx, ny, nz, npml, steps, seed, nfreq):
    d = 5e-9
    dk = decks.Deck(nx, ny, nz, d, d, d, media=[(1.0, 1.0, 0.0, 0.0)] * 3)
    _spheres(dk, [c for c in decks.jittered_lattice((nx, ny, nz), 40.0, 3.0, seed)
                  if all(npml + 24 <= v <= n - npml - 24 for v, n in zip(c, (nx, ny, nz)))], 15.0, 2)
    inset = npml + 8
    dk.pml = decks.pml_params(npml)
    lam, tau = 550e-9, 2e-15
    dk.n0 = int(4 * lam / C0 / dk.dt)  # the pulse is about to enter the box
    dk.tfsf = {"lambda": lam, "dlambda": decks.dlambda_for_tau(lam, tau), "w0": 400e-9 * min(nx, ny, nz) / 256.0,
               "z0_deck": 0.0, "xs": (nx / 2 + 0.5) * d, "ys": (ny / 2 + 0.5) * d, "zs": 0.0, "k0": nz // 2,
               "theta": 30.0, "phi": 45.0, "E0": 1.0, "psi": 0.0, "n6": [inset] * 6, "Nt": dk.n0 + 8 * steps,
               "cwmode": 0}
    freqs = np.linspace(0.8, 1.2, nfreq) * C0 / lam
    lo, hi = inset - 2, [n - inset + 2 for n in (nx, ny, nz)]
    for a, axis in enumerate("xyz"):
        mask = 0x3F & ~((1 << a) | (1 << (3 + a)))  # the tangential components
        wa, ha = {0: (1, 2), 1: (0, 2), 2: (0, 1)}[a]
        for pos in (lo, hi[a]):
            dk.ports.append(decks.Port("plain", dict(dir=axis, position=(pos + 0.5) * d, w1=(lo + 0.5) * d,
                                                     w2=(hi[wa] + 0.5) * d, h1=(lo + 0.5) * d,
                                                     h2=(hi[ha] + 0.5) * d), dft_freqs=freqs, dft_mask=mask))
    dk.dl = decks.dl_params_metal()
    return dk


def _laser(nx, ny, nz, npml, steps, seed, nfreq):
    dk = decks.config4_member(nx, ny, nz, seed, steps=steps, nfreq=nfreq, npml=npml, port=False)
    dk.sources = [(c, i, j, k, _wave(dk, steps)) for c, i, j, k, _ in dk.sources]
    c = (nx // 2 + 0.5, ny // 2 + 0.5, nz // 2 + 0.5)
    dk.ports = [decks.Port("spherical", dict(r=0.39 * min(nx, ny, nz) * dk.dx, xc=c[0] * dk.dx, yc=c[1] * dk.dx,
                                             zc=c[2] * dk.dx, theta1=0.0, theta2=180.0, phi1=0.0, phi2=360.0),
                           dft_freqs=np.linspace(0.9, 1.1, nfreq) * C0 / 600e-9)]
    return dk


def _decks(case, seed):
    """The decks of a case: one, or one per member or job."""
    k, nf = case["kind"], case["nfreq"]
    a = (case["nx"], case["ny"], case["nz"], case["npml"], case["steps"])
    if k == "scatterer":
        return [_scatterer(*a, seed)]
    if k == "dispersive":
        return [_dispersive(*a, seed, nf)]
    if k == "laser":
        return [_laser(*a, seed, nf)]
    # nx..ny: range of edges, nz: how many; the shapes belong to the case, the disorder to the seed
    rng = np.random.Generator(np.random.PCG64(case["nx"] * 1000 + case["nz"]))
    out = []
    for m in range(case["nz"]):
        e = [int(v) for v in rng.integers(case["nx"], case["ny"] + 1, size=3)]
        if k == "ensemble":
            out.append(_laser(*e, case["npml"], case["steps"], seed * 100 + m, nf))
            continue
        steps = int(case["steps"] * (0.5 + m / case["nz"]))
        make = (lambda *q: _scatterer(*q), lambda *q: _dispersive(*q, nf), lambda *q: _laser(*q, nf))[m % 3]
        out.append(make(*e, case["npml"], steps, seed * 100 + m))
        out[-1].nsteps = steps
    return out


def _modes(case, shape3, npml, seed):
    """A developed field: for each E component a few standing waves of 12 to 40
    cells, zero in the CPML, as per-axis factors."""
    rng = np.random.Generator(np.random.PCG64(seed + 77))
    out = []
    for _ in range(3):
        comp = []
        for _ in range(3):
            axes = []
            for n in shape3:
                x = np.arange(n, dtype=np.float64)
                lo, hi = npml + 2, n - 1 - npml - 2
                w = np.where((x > lo) & (x < hi), np.sin(PI * np.clip((x - lo) / (hi - lo), 0, 1)) ** 2, 0.0)
                axes.append(w * np.cos(2 * PI * x / rng.uniform(12, 40) + rng.uniform(0, 2 * PI)))
            comp.append((rng.uniform(0.3, 1.0), axes))
        out.append(comp)
    return out


def _field_of(comp, dev):
    v = None
    for amp, axes in comp:
        x, y, z = (torch.from_numpy(q).to(dev) for q in axes)
        t = (amp * x)[:, None, None] * y[None, :, None] * z[None, None, :]
        v = t if v is None else v + t
    return v


# ----------------------------------------------------------------- prepare

def _prec(case):
    return cps.FP32 if case["dtype"] == "f32" else cps.FP64


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=torch.cuda.is_available())


class _Reader:
    """Reads a grid's results into buffers that are kept: pinned FP64 staging
    as the library writes it, FP32 results for FP32 grids."""

    def __init__(self, g, comps, f32, stage):
        self.g, self.comps, self.stage = g, comps, stage
        dt = torch.float32 if f32 else torch.float64
        self.f32 = f32
        self.ports = [p for p in range(len(g.ports)) if g.ports[p][2]]
        size = lambda p: (g.ports[p][1], g.ports[p][2], 2, g.ports[p][0])  # noqa: E731
        make = (lambda s: torch.empty(s, dtype=dt)) if f32 else (lambda s: _pinned(s, dt))
        self.fields = [make(g.shape3) for _ in comps]
        self.dft = [make(size(p)) for p in self.ports]

    def values(self):
        return max([f.numel() for f in self.fields + self.dft], default=0)

    def read(self):
        for c, out in zip(self.comps, self.fields):
            to = self.stage[:out.numel()].view(out.shape) if self.f32 else out
            code = cps.lib().cps_field_download(self.g.h, c, ctypes.cast(to.data_ptr(),
                                                                         ctypes.POINTER(ctypes.c_double)))
            if code:
                raise cps.CpsError(code, cps.lib().cps_last_error().decode())
            if self.f32:
                out.copy_(to)
        for p, out in zip(self.ports, self.dft):
            to = self.stage[:out.numel()].view(out.shape) if self.f32 else out
            self.g.port_dft(p, raw=True, out=to.numpy())
            if self.f32:
                out.copy_(to)
        return {"fields": self.fields, "dft": self.dft}


def _comps(case):
    return {ALL: list(range(6)), EZ: [2], "ports": []}[case["read"]]


def prepare(case, seed):
    dks = _decks(case, seed)
    if case["kind"] == "served":
        return {"server": cps.Server(_prec(case), max_jobs=8, budget_bytes=16 * 10 ** 9), "decks": dks,
                "points": [[cps.port_points(dk, p) for p in dk.ports] for dk in dks]}
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    batch = cps.Batch(_prec(case)) if case["kind"] == "ensemble" else None
    grids = []
    for dk in dks:
        g = cps.Grid.from_deck(dk, _prec(case))
        for c, comp in enumerate(_modes(case, g.shape3, case["npml"], seed)):
            g.set_field(c, _field_of(comp, dev).cpu().numpy())
        if case["path"] == "calls":
            g.set_record(True)
        if batch is not None:
            batch.add(g)
        grids.append(g)
    readers = [_Reader(g, _comps(case), case["dtype"] == "f32", None) for g in grids]
    if case["dtype"] == "f32":  # one staging buffer for the program's read-outs
        stage = _pinned(max(r.values() for r in readers), torch.float64)
        for r in readers:
            r.stage = stage
    return {"batch": batch, "grids": grids, "readers": readers, "steps": case["steps"], "path": case["path"]}


# --------------------------------------------------------------------- run

def _main_loop(g, steps):
    """The reference's loop body, one call per routine."""
    n = g.get_step()
    for n in range(n, n + steps):
        g.op("h_bulk")
        g.op("tfsf_h", n, 0x3F)
        g.op("h_pml")
        g.op("e_bulk")
        g.op("dl")
        g.op("tfsf_e", n, 0x3F)
        g.op("e_pml")
        for p in range(len(g.ports)):
            g.op("port_sample", p, n)
    g.set_step(n + 1)


def _serve(state):
    """Every job through the server: grid from the deck, its steps, its spectra
    (a job without a port DFT: its Ez)."""
    dks, got = state["decks"], [None] * len(state["decks"])

    def build(m):
        return lambda: cps.Grid.from_deck(dks[m], cps.FP32, port_points_list=state["points"][m])

    def done(m):
        def read(g, status):
            if status == 0:
                r = [g.port_dft(p, raw=True) for p in range(len(g.ports)) if g.ports[p][2]] or [g.field(2)]
                got[m] = [torch.from_numpy(v).float() for v in r]
        return read

    for m, dk in enumerate(dks):
        state["server"].submit(build(m), done(m), dk.nsteps, cps.footprint(dk))
    state["server"].drain()
    return {"jobs": got}


def run(state):
    if "server" in state:
        return _serve(state)
    if state["batch"] is not None:
        state["batch"].step(state["steps"])
    else:
        g = state["grids"][0]
        if state["path"] == "calls":
            _main_loop(g, state["steps"])
        else:
            g.step(state["steps"], cps.PLAIN if state["path"] == "plain" else cps.FUSED)
    return {"grids": [r.read() for r in state["readers"]]}


# -------------------------------------------------------------------- work

def work(case):
    """Per time step: each field word read and written once and each ID read
    once; two psi words per side and CPML cell; the dispersive or gain state
    words of its cells, read and written once.  Per pass: the results.  FP64
    words are twice as long.  Operations: the Yee curls, psi, and the state
    updates of each cell."""
    w = 4 if case["dtype"] == "f32" else 8

    def grid(kind, nx, ny, nz, steps):
        cells, npml = nx * ny * nz, case["npml"]
        slab = sum(2 * npml * cells / n for n in (nx, ny, nz))
        words, flops = 12 * cells + 8 * slab, 36 * cells + 24 * slab
        if kind == "dispersive":
            m = 1
            for n in (nx, ny, nz):
                q = max(1, int(n // 40.0))
                at = (n - (q - 1) * 40.0) / 2.0 + 40.0 * np.arange(q)
                m *= int(((at >= npml + 24) & (at <= n - npml - 24)).sum())
            dl = m * 4.0 / 3.0 * PI * 15.0 ** 3
            words, flops = words + 2 * 18 * dl, flops + 100 * dl
        if kind == "laser":
            gain = 0.92 * cells
            words, flops = words + 2 * 15 * gain, flops + 90 * gain
        return steps * (words * w + cells), steps * flops

    def results(kind, nx, ny, nz, field):
        n = field * (nx + 1) * (ny + 1) * (nz + 1)
        if kind == "laser":
            n += 19.8 * (0.39 * min(nx, ny, nz)) ** 2 * 6 * case["nfreq"] * 2
        if kind == "dispersive":
            q = 2 * (case["npml"] + 6) - 1
            n += 2 * sum((a - q) * (b - q) for a, b in ((nx, ny), (ny, nz), (nx, nz))) * 4 * case["nfreq"] * 2
        return n * w

    nbytes = flops = 0.0
    if case["kind"] in ("ensemble", "served"):
        rng = np.random.Generator(np.random.PCG64(case["nx"] * 1000 + case["nz"]))
        for m in range(case["nz"]):
            e = [int(v) for v in rng.integers(case["nx"], case["ny"] + 1, size=3)]
            kind, steps = "laser", case["steps"]
            if case["kind"] == "served":
                kind, steps = ("scatterer", "dispersive", "laser")[m % 3], int(steps * (0.5 + m / case["nz"]))
            b, f = grid(kind, *e, steps)
            nbytes += b + results(kind, *e, 1 if kind == "scatterer" else 0)
            flops += f
    else:
        e = (case["nx"], case["ny"], case["nz"])
        nbytes, flops = grid(case["kind"], *e, case["steps"])
        nbytes += results(case["kind"], *e, len(_comps(case)))
    return {"bytes": float(nbytes), "flops": float(flops)}


# ------------------------------------------------------------------- exact

def _grading(np_, first, half, dt, delta, p):
    """kappa, b, c of one CPML end: on E planes (half = 0, np + 1 of them) or
    H planes (half = 0.5, np of them)."""
    q = np.arange(np_ + 1 if half == 0 else np_, dtype=np.float64)
    near, far = (np_ - q - half) / np_, (q + half) / np_
    ps, pa = (near ** p["m"], far ** p["malp"]) if first else (far ** p["m"], near ** p["malp"])
    smax = p["sig_ratio"] * 0.8 * (p["m"] + 1) / (delta * math.sqrt(MU0 / EPS0))
    sig, kap, alp = smax * ps, 1.0 + (p["kapmax"] - 1.0) * ps, p["alpmax"] * pa
    b = np.exp(-(sig / kap + alp) * dt / EPS0)
    den = sig + kap * alp
    c = np.where(den > 0, sig * (b - 1.0) / np.where(den > 0, den, 1.0) / kap / delta, 0.0)
    return kap, b, c


class _Exact:
    """The time-stepping loop in FP64 torch, arrays [i][j][k] of (n + 1)^3."""

    def __init__(self, dk, dev):
        self.dk, self.dev = dk, dev
        self.n = (dk.nx, dk.ny, dk.nz)
        self.dx = (dk.dx, dk.dy, dk.dz)
        self.dt = dt = dk.dt
        t = lambda v: torch.as_tensor(np.asarray(v), dtype=torch.float64, device=dev)  # noqa: E731
        self.E = [torch.zeros(dk.shape3, dtype=torch.float64, device=dev) for _ in range(3)]
        self.H = [torch.zeros(dk.shape3, dtype=torch.float64, device=dev) for _ in range(3)]
        eps, mu, sig, sigm = np.array(dk.media, dtype=np.float64).T
        tab = [(2 * EPS0 * eps - sig * dt) / (2 * EPS0 * eps + sig * dt), 2 * dt / (2 * EPS0 * eps + sig * dt),
               (2 * MU0 * mu - sigm * dt) / (2 * MU0 * mu + sigm * dt), 2 * dt / (2 * MU0 * mu + sigm * dt)]
        ids = torch.from_numpy(dk.ids).to(dev)
        self.inner = tuple(slice(1, n) for n in self.n)
        self.low = tuple(slice(0, n) for n in self.n)
        ie, ih = ids[self.inner].long(), ids[self.low].long()
        self.aE, self.bE = t(tab[0])[ie], t(tab[1])[ie]
        self.aH, self.bH = t(tab[2])[ih], t(tab[3])[ih]
        self.ce = self.bE
        self._pml(t)
        self.dl = self.gain = self.beam = None
        if dk.dl:
            self._dl_init(ie)
        if dk.gain:
            self._gain_init(ie)
        if dk.tfsf:
            self._beam_init(t)
        self.step = dk.n0
        self.src = [(c, i, j, k, np.asarray(w)) for c, i, j, k, w in dk.sources]

    # one-sided differences of a component over the update range
    def dE(self, c, a):
        up = tuple(slice(1, n + 1) if b == a else slice(0, n) for b, n in enumerate(self.n))
        return self.E[c][up] - self.E[c][self.low]

    def dH(self, c, a):
        dn = tuple(slice(0, n - 1) if b == a else slice(1, n) for b, n in enumerate(self.n))
        return self.H[c][self.inner] - self.H[c][dn]

    def _pml(self, t):
        self.sE, self.sH, self.slabs = [], [], []
        p = self.dk.pml
        for a, n in enumerate(self.n):
            np_, d = p["npml"][2 * a], self.dx[a]
            se, sh = np.full(n, 1.0 / d), np.full(n, 1.0 / d)
            for first in (True, False):
                kap, b, c = _grading(np_, first, 0, self.dt, d, p)
                kh, bh, ch = _grading(np_, first, 0.5, self.dt, d, p)
                lo = 0 if first else n - np_
                if first:
                    se[:np_ + 1] /= kap
                    be, ce, at = b[1:], c[1:], slice(0, np_)  # planes 1..np, counted from 1
                else:
                    se[lo:] /= kap[:np_]
                    be, ce, at = b[:np_], c[:np_], slice(lo - 1, n - 1)
                sh[lo:lo + np_] /= kh
                self.slabs.append((a, at, slice(lo, lo + np_), self._on(t(be), a), self._on(t(ce), a),
                                   self._on(t(bh), a), self._on(t(ch), a), [0.0] * 4))
            self.sE.append(self._on(t(se[1:]), a))
            self.sH.append(self._on(t(sh), a))

    @staticmethod
    def _on(v, a):
        return v.view([-1 if b == a else 1 for b in range(3)])

    def _h(self):
        E, H = self.E, self.H
        d = {(c, a): self.dE(c, a) for c in range(3) for a in range(3) if a != c}
        for c in range(3):
            u, v = (c + 1) % 3, (c + 2) % 3  # H_c += b (dE_u/dv - dE_v/du)
            h = H[c][self.low]
            h.copy_(self.aH * h + self.bH * (d[u, v] * self.sH[v] - d[v, u] * self.sH[u]))
        self._apply_beam(True)
        for a, _, at, _, _, b, c, psi in self.slabs:
            cut = tuple(at if q == a else slice(None) for q in range(3))
            u, v = (a + 1) % 3, (a + 2) % 3
            s = 1.0 if a == 0 else -1.0  # the signs of the reference's H-side CPML (CPML.cpp:617-682)
            for q, (dst, src, sgn) in enumerate(((u, v, s), (v, u, -s))):
                psi[2 + q] = b * psi[2 + q] + c * d[src, a][cut]
                H[dst][self.low][cut].add_(psi[2 + q] * self.bH[cut], alpha=sgn)

    def _e(self):
        E, H = self.E, self.H
        d = {(c, a): self.dH(c, a) for c in range(3) for a in range(3) if a != c}
        curl = []
        for c in range(3):
            u, v = (c + 1) % 3, (c + 2) % 3  # E_c += b (dH_v/du - dH_u/dv)
            curl.append(d[v, u] * self.sE[u] - d[u, v] * self.sE[v])
        if self.dl:
            old = [e[self.inner][self.dl_at] for e in E]
        for c in range(3):
            e = E[c][self.inner]
            e.copy_(self.aE * e + self.bE * curl[c])
        if self.dl:
            for c in range(3):
                E[c][self.inner][self.dl_at] = self._dl(c, old[c], curl[c][self.dl_at])
        if self.gain:
            self._gain()
        self._apply_beam(False)
        for c, i, j, k, w in self.src:
            if 0 <= self.step < len(w):
                E[c][i, j, k] += float(w[self.step])
        for a, at, _, b, c, _, _, psi in self.slabs:
            cut = tuple(at if q == a else slice(None) for q in range(3))
            u, v = (a + 1) % 3, (a + 2) % 3
            for q, (dst, src, sgn) in enumerate(((u, v, -1.0), (v, u, 1.0))):
                psi[q] = b * psi[q] + c * d[src, a][cut]
                E[dst][self.inner][cut].add_(psi[q] * self.ce[cut], alpha=sgn)

    # Drude-Lorentz cells: one Drude or Lorentz current per pole and component
    def _dl_init(self, ie):
        p, dt = self.dk.dl, self.dt
        kap, beta, alpha, xi, gam = [], [], [], [], []
        for f, g in zip(p["fD"], p["gD"]):
            w, g = 2 * PI * f, 2 * PI * g
            kap.append((1 - g * dt / 2) / (1 + g * dt / 2))
            beta.append(w * w * EPS0 * dt / 2 / (1 + g * dt / 2))
        for f, dl, de in zip(p["fL"], p["dL"], p["depsL"]):
            w, dl = 2 * PI * f, 2 * PI * dl
            alpha.append((2 - w * w * dt * dt) / (1 + dl * dt))
            xi.append((dl * dt - 1) / (1 + dl * dt))
            gam.append(EPS0 * de * w * w * dt * dt / (1 + dl * dt))
        den = 2 * EPS0 * p["epsInf"] + p["sigma"] * dt + dt * sum(beta) + sum(gam) / 2
        self.dl = dict(kap=kap, beta=beta, alpha=alpha, xi=xi, gam=gam, C2=sum(gam) / 2 / den, C3=2 * dt / den,
                       C1=(2 * EPS0 * p["epsInf"] - p["sigma"] * dt - dt * sum(beta)) / den,
                       C4=[(1 + k) * dt / den for k in kap], C5=[(1 + a) * dt / den for a in alpha],
                       C6=[x * dt / den for x in xi])
        self.dl_at = (ie == 2).nonzero(as_tuple=True)
        self.ce = torch.where(ie == 2, self.dl["C3"], self.bE)
        z = lambda: torch.zeros(len(self.dl_at[0]), dtype=torch.float64, device=self.dev)  # noqa: E731
        self.dl_state = [dict(JD=[z() for _ in kap], JL=[z() for _ in alpha], JL1=[z() for _ in alpha], E1=z())
                         for _ in range(3)]

    def _dl(self, c, e, curl):
        D, s = self.dl, self.dl_state[c]
        new = D["C1"] * e + D["C2"] * s["E1"] + D["C3"] * curl
        for q, j in enumerate(s["JD"]):
            new = new - D["C4"][q] * j
        for q, j in enumerate(s["JL"]):
            new = new - D["C5"][q] * j - D["C6"][q] * s["JL1"][q]
        for q, j in enumerate(s["JD"]):
            s["JD"][q] = D["kap"][q] * j + D["beta"][q] * (new + e)
        for q, j in enumerate(s["JL"]):
            s["JL"][q] = D["alpha"][q] * j + D["xi"][q] * s["JL1"][q] + D["gam"][q] * (new - s["E1"]) / 2 / self.dt
            s["JL1"][q] = j
        s["E1"] = e
        return new

    # four-level gain: two polarisations and four populations per cell
    def _gain_init(self, ie):
        p, dt = self.dk.gain, self.dt
        wa, wb = 2 * PI * C0 / p["lambda_a"], 2 * PI * C0 / p["lambda_b"]
        g = {}
        for s, w, t in (("a", wa, p["t21"]), ("b", wb, p["t30"])):
            q = 1 + p["gamma_" + s] * dt / 2
            g[s] = ((2 - w * w * dt * dt) / q, (p["gamma_" + s] * dt / 2 - 1) / q,
                    dt * dt * 6 * PI * EPS0 * C0 ** 3 / (w * w * t) / q)
        g["CEP"] = 2 * p["N_0"] * self.dx[0] * self.dx[1] * self.dx[0] / EPS0 / dt
        g["ha"], g["hb"] = H_PLANCK * wa * dt / 2 / PI, H_PLANCK * wb * dt / 2 / PI
        self.gain = g
        self.gain_on = ie == p.get("gain_id", 5)
        z = lambda v=0.0: torch.full_like(self.bE, v)  # noqa: E731
        self.P = [{s: (z(), z()) for s in "ab"} for _ in range(3)]
        self.N = [z(1.0), z(1.0), z(), z()]

    def _gain(self):
        g, p, dt, N = self.gain, self.dk.gain, self.dt, self.N
        dN = {"a": N[2] - N[1], "b": N[3] - N[0]}
        sa = sb = s2 = 0.0
        for c in range(3):
            e = self.E[c][self.inner]
            e1 = e.clone()
            dP = {}
            for s in "ab":
                now, was = self.P[c][s]
                new = g[s][0] * now + g[s][1] * was + g[s][2] * dN[s] * e1
                dP[s] = (new - now, new - was)
                self.P[c][s] = (new, now)
            e.sub_(torch.where(self.gain_on, g["CEP"] * (dP["a"][0] + dP["b"][0]), 0.0))
            sa = sa + e1 * dP["a"][1]
            sb = sb + e1 * dP["b"][1]
            s2 = s2 + (e + e1) * (dP["a"][0] if c == 1 else dP["a"][1])
        t30, t32, t21, t10 = p["t30"], p["t32"], p["t21"], p["t10"]
        N0 = N[0]
        N3 = t30 * t32 * dt / (2 * t30 * t32 + t30 * dt * (1 - N[2]) + t32 * dt * (1 - N0)) * \
            (N[3] * ((N0 - 1) / t30 + (N[2] - 1) / t32 + 2 / dt) + sb / g["hb"]) + p.get("pump", 0.0) * dt * N0
        N1 = t10 * t21 * dt / (2 * t10 * t21 + t10 * dt * N[2] + t21 * dt * (1 - N0)) * \
            (N[1] * ((N0 - 1) / t10 - N[2] / t21 + 2 / dt) + N[2] / (t21 / 2) - sa / g["ha"])
        N2 = t32 * t21 * dt / (2 * t32 * t21 + t21 * dt * N3 + t32 * dt * (1 - N1)) * \
            (N[2] * ((N1 - 1) / t21 - N3 / t32 + 2 / dt) + N3 / (t32 / 2) + s2 / g["ha"])
        self.N = [2.0 - N1 - N2 - N3, N1, N2, N3]

    # TF/SF Gaussian beam: per face and component a strip of cells, its delays and profile
    def _beam_init(self, t):
        q, dt = self.dk.tfsf_abi(), self.dt
        th, ph, ps = (math.radians(q[k]) for k in ("theta", "phi", "psi"))
        E0, eta = q["E0"], math.sqrt(MU0 / EPS0)
        Ei = (E0 * (math.cos(ps) * math.sin(ph) - math.sin(ps) * math.cos(th) * math.cos(ph)),
              E0 * (-math.cos(ps) * math.cos(ph) - math.sin(ps) * math.cos(th) * math.sin(ph)),
              E0 * math.sin(ps) * math.sin(th))
        Hi = (E0 / eta * (math.sin(ps) * math.sin(ph) + math.cos(ps) * math.cos(th) * math.cos(ph)),
              E0 / eta * (-math.sin(ps) * math.cos(ph) + math.cos(ps) * math.cos(th) * math.sin(ph)),
              -E0 / eta * math.cos(ps) * math.sin(th))
        k = np.array([math.sin(th) * math.cos(ph), math.sin(th) * math.sin(ph), math.cos(th)])
        org = (q["i0"], q["j0"], q["k0"])
        lo = [q["n6"][2 * a] for a in range(3)]
        hi = [self.n[a] - q["n6"][2 * a + 1] for a in range(3)]
        l0 = min(sum(k[a] * ((lo, hi)[(m >> a) & 1][a] - org[a]) * self.dx[a] for a in range(3)) / C0
                 for m in range(8))
        zr = PI * q["w0"] ** 2 / q["lambda_"]
        nu = C0 / q["lambda_"]
        dnu = C0 / (q["lambda_"] - q["dlambda"] / 2) - C0 / (q["lambda_"] + q["dlambda"] / 2)
        sig, t0 = (2 * PI * dnu) ** 2 / (16 * math.log(2)), 5 / nu
        tt = np.arange(q["Nt"] + 1) * dt - t0
        pulse = lambda x: np.exp(-sig * x * x) * np.sin(2 * PI * nu * x)  # noqa: E731
        pad = lambda v: t(np.concatenate([v, np.zeros(2)]))  # noqa: E731
        self.Nt, self.beam, self.inc = q["Nt"], {True: [], False: []}, {True: pad(pulse(tt)),
                                                                         False: pad(pulse(tt + dt / 2))}
        for isH in (False, True):
            inc, cst = (Ei, MU0) if isH else (Hi, EPS0)
            for a in (1, 0, 2):
                u, v = [b for b in range(3) if b != a]
                for far in (0, 1):
                    at = (lo, hi)[far][a]
                    off = 0.0 if isH else (0.5 if far else -0.5)
                    for which in (0, 1):
                        # which tangential axis the strip is short along, and the corrected component
                        comp = (v if which == 0 else u) if isH else (u if which == 0 else v)
                        other = u + v - comp
                        ue, ve = (hi[u], hi[v] + 1) if which == 0 else (hi[u] + 1, hi[v])
                        if isH and a == 0:
                            ue, ve = hi[u], hi[v]
                        # the sign of the curl term the strip makes up for
                        s = (1.0 if (comp - a) % 3 == 1 else -1.0) * (-1.0 if isH else 1.0) * (-1.0 if far else 1.0)
                        coef = s * dt / (cst * self.dx[a]) * inc[other]
                        pos = [None] * 3
                        pos[a] = np.array([(at - org[a] + off) * self.dx[a]])
                        pos[u] = (np.arange(lo[u], ue) - org[u]) * self.dx[u]
                        pos[v] = (np.arange(lo[v], ve) - org[v]) * self.dx[v]
                        x, y, z = (pos[b].reshape([-1 if w == b else 1 for w in range(3)]) for b in range(3))
                        rk = x * k[0] + y * k[1] + z * k[2]
                        rho2 = x * x + y * y + z * z - rk * rk
                        wz2 = q["w0"] ** 2 * (1 + (rk - q["z0"]) ** 2 / zr ** 2)
                        plane = at + ((1 if far else -1) if isH else 0)
                        cut = [None] * 3
                        cut[a] = slice(plane, plane + 1)
                        cut[u], cut[v] = slice(lo[u], ue), slice(lo[v], ve)
                        self.beam[isH].append((comp, tuple(cut), t((rk / C0 - l0) / dt),
                                               t(coef * np.exp(-rho2 / wz2))))

    def _apply_beam(self, isH):
        if self.beam is None:
            return
        tab = self.inc[isH]
        for comp, cut, delay, prof in self.beam[isH]:
            r = self.step - delay
            f = torch.floor(r)
            m = f.long().clamp(0, self.Nt + 1)
            v = (1 - (r - f)) * tab[m] + (r - f) * tab[(m + 1).clamp(max=self.Nt + 2)]
            (self.H if isH else self.E)[comp][cut].add_(torch.where(r > 0, v, 0.0) * prof)

    def run(self, steps, ports):
        """Steps the loop; the DFT of each port [ncomp][nfreq][2][npts]."""
        flat = [torch.from_numpy(np.ascontiguousarray(pts)).to(self.dev).long() for _, pts in ports]
        seen = [[[] for c in range(6) if p.dft_mask >> c & 1] for p, _ in ports]
        first = self.step
        for _ in range(steps):
            self._h()
            self._e()
            F = self.E + self.H
            for (p, _), at, s in zip(ports, flat, seen):
                for q, c in enumerate(c for c in range(6) if p.dft_mask >> c & 1):
                    s[q].append(F[c][at[:, 0], at[:, 1], at[:, 2]])
            self.step += 1
        out = []
        n = np.arange(first, first + steps, dtype=np.float64)
        for (p, _), s in zip(ports, seen):
            acc = []
            for q, c in enumerate(c for c in range(6) if p.dft_mask >> c & 1):
                ph = 2 * PI * np.asarray(p.dft_freqs)[:, None] * ((n if c < 3 else n - 0.5) * self.dt)[None, :]
                x = torch.stack(s[q])
                s[q] = None
                w = [torch.from_numpy(v).to(self.dev) for v in (np.cos(ph), -np.sin(ph))]
                acc.append(torch.stack([w[0] @ x, w[1] @ x], dim=1))
            out.append(torch.stack(acc))
        return out


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    out = []
    for dk in _decks(case, seed):
        x = _Exact(dk, dev)
        if case["kind"] != "served":
            for c, comp in enumerate(_modes(case, dk.shape3, case["npml"], seed)):
                x.E[c].copy_(_field_of(comp, dev))
        ports = [(p, cps.port_points(dk, p)) for p in dk.ports if p.dft_freqs is not None]
        dft = x.run(dk.nsteps if case["kind"] == "served" else case["steps"], ports)
        if case["kind"] == "served":
            out.append(dft or [x.E[2]])
        else:
            out.append({"fields": [(x.E + x.H)[c] for c in _comps(case)], "dft": dft})
        del x
    return {"jobs": out} if case["kind"] == "served" else {"grids": out}
