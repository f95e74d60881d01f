"""Performance cases of the step engine: what a program that uses it has it do.

A pass is the way every run of the engine goes: primitives come up from
page-locked host memory (a restart, or a setup's initial data), the grid takes
its steps on the device, and the primitives come down for a dump.  Grids,
boundaries and options are the setups' own: the Balsara-1 shock tube, the
advected field loop, the periodic linear wave, the magnetised torus, the
circumbinary disk, and a server's batch of small grids.  FP64 and the mixed
form; the form with fused multiply-adds is measured on the torus.

prepare() makes inputs and a resident grid, run() is one pass, exact() the
same steps in plain torch at 64 bits for the Minkowski problems.
"""
import math

import numpy as np
import torch

import coolharm3d_b200 as hg
from coolharm3d_b200 import pnbbh, setups, torus

NG = hg.NG
PREC = {"fp64": hg.PREC_FP64, "mixed": hg.PREC_MIXED, "fma": hg.PREC_FP64_FMA}


def listed():
    return [
        # the smallest grids: a 1D shock tube and the server's smallest 3D wave, where launches count
        dict(name="tube_1024", kind="tube", n1=1024, n2=1, n3=1, prec="fp64", steps=40),
        dict(name="wave_32", kind="wave", n1=32, n2=32, n3=32, prec="fp64", steps=20),
        # 2D: one direction has a single zone
        dict(name="loop_256", kind="loop", n1=256, n2=256, n3=1, prec="fp64", steps=20),
        # the server's batch: a dozen small grids advanced together
        dict(name="batch_12", kind="batch", members=12, size=1.0, prec="fp64", steps=20),
        # the linear wave at the server's largest size and at the convergence study's; the mixed form
        dict(name="wave_128", kind="wave", n1=128, n2=128, n3=128, prec="fp64", steps=10),
        dict(name="wave_128_mixed", kind="wave", n1=128, n2=128, n3=128, prec="mixed", steps=10),
        dict(name="wave_256", kind="wave", n1=256, n2=256, n3=256, prec="fp64", steps=10),
        # the torus: a rank's block of it, an odd-sized one, and the production grid in both forms
        dict(name="torus_96", kind="torus", n1=96, n2=96, n3=64, prec="fp64", steps=20),
        dict(name="torus_131_odd", kind="torus", n1=131, n2=77, n3=37, prec="fma", steps=20),
        dict(name="torus_192", kind="torus", n1=192, n2=192, n3=128, prec="fp64", steps=20),
        dict(name="torus_192_mixed", kind="torus", n1=192, n2=192, n3=128, prec="mixed", steps=20),
        # the binary's circumbinary disk: the metric evaluated on the device every step
        dict(name="disk_75", kind="disk", n1=75, n2=40, n3=100, prec="fp64", steps=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    # the tube and the loop have even sizes only: the zone in the middle of an
    # odd one lies at radius 0, where the setups' floors are infinite
    kind = rng.choice(["tube", "loop", "wave", "wave", "torus", "torus", "disk", "batch"])
    prec = rng.choice(["fp64", "fp64", "mixed"])
    if kind == "tube":
        return dict(kind=kind, n1=2 * _log(rng, 250, 2500), n2=1, n3=1, prec=prec, steps=rng.randint(20, 60))
    if kind == "loop":
        return dict(kind=kind, n1=2 * _log(rng, 48, 260), n2=2 * _log(rng, 48, 260), n3=1, prec=prec, steps=rng.randint(10, 30))
    if kind == "wave":
        return dict(kind=kind, n1=_log(rng, 24, 180), n2=_log(rng, 24, 180), n3=_log(rng, 24, 180), prec=prec,
                    steps=rng.randint(5, 15))
    if kind == "torus":
        return dict(kind=kind, n1=_log(rng, 48, 192), n2=_log(rng, 40, 160), n3=_log(rng, 16, 128), prec=prec,
                    steps=rng.randint(10, 20))
    if kind == "disk":
        return dict(kind=kind, n1=_log(rng, 48, 90), n2=_log(rng, 24, 64), n3=_log(rng, 32, 100), prec="fp64",
                    steps=rng.randint(5, 12))
    return dict(kind=kind, members=rng.randint(3, 16), size=rng.uniform(0.5, 1.5), prec=prec, steps=rng.randint(10, 25))


# --------------------------------------------------------------------------
# inputs

def _ghosts(p, n, bc):
    """Ghost zones of the Minkowski setups: wrapped, or copies of the nearest zone."""
    for a, m in enumerate(n):
        x = np.arange(m + 2 * NG) - NG
        src = NG + (np.clip(x, 0, m - 1) if bc == hg.BC_CARTESIAN_OUTFLOW else x % m)
        p = np.take(p, src, axis=a)
    return p


def _minkowski(kind, n, prec, seed):
    """(Problem, primitives with ghosts, first time step) of one Minkowski setup."""
    rng = np.random.default_rng(seed)
    if kind == "tube":
        prob = setups.balsara1(n[0], precision=prec)
        s = slice(NG, NG + n[0])
        left = prob.p_init[s, NG, NG, 6] > 0
        for side in (left, ~left):  # states within 10% of the test's own
            for l in (0, 1, 6):
                prob.p_init[s, NG, NG, l][side] *= rng.uniform(0.9, 1.1)
    elif kind == "loop":
        prob = setups.field_loop(n, v0=float(rng.uniform(0.3, 0.6)), precision=prec)
    else:
        mode = ("fast", "alfven", "slow")[int(rng.integers(3))]
        prob = setups.linear_wave_3d(n, mode=mode, amp=10.0 ** rng.uniform(-6, -3), precision=prec)
        sl = tuple(slice(NG, NG + m) for m in n)
        prob.p_init[sl] = np.roll(prob.p_init[sl], int(rng.integers(1, n[0])), axis=0)
    prob.desc.grid_length[0] = 1e9  # away from the final time
    dt = 0.25 * prob.desc.cour * min(prob.desc.dx[a + 1] for a in range(3) if n[a] > 1)
    return prob, _ghosts(prob.p_init, n, prob.desc.bc_type), dt


def _members(case, seed):
    """(kind, n, seed) of a batch's grids, the server's mix of kinds and sizes."""
    sizes = {"tube": (512, 1024, 2048), "loop": (96, 128, 192), "wave": (24, 32, 48)}
    out = []
    for m in range(case["members"]):
        kind = ("tube", "loop", "wave")[m % 3]
        s = 2 * max(8, int(sizes[kind][m // 3 % 3] * case["size"] / 2))
        out.append((kind, {"tube": (s, 1, 1), "loop": (s, s, 1), "wave": (s, s, s)}[kind], seed * 1000 + m))
    return out


def _pinned(p):
    buf = hg.pinned_array(p.shape)
    buf[...] = p
    return buf


class Grid:
    """A resident grid with its start (primitives, t, dx[0]) and a host buffer for its dumps."""

    def __init__(self, desc, p, t, dt):
        self.engine = hg.Engine(desc)
        self.p, self.t, self.dt = _pinned(p), t, dt
        self.out = hg.pinned_array(p.shape)

    def load(self):
        self.engine.upload(self.p)
        self.engine.set_time(self.t, self.dt)


def _minkowski_grid(kind, n, prec, seed):
    prob, p, dt = _minkowski(kind, n, PREC[prec], seed)
    g = Grid(prob.desc, p, 0.0, dt)
    g.engine.set_geometry(prob.geom)
    g.engine.set_cell_data(prob.cell6)
    return g


def _torus_engine(n, prec):
    desc = torus.torus_desc(n, precision=PREC[prec])
    tab = torus.torus_tables(desc)
    return desc, tab, lambda e: (e.set_geometry(tab["geom"], tab["conn"]), e.set_cell_data(tab["cell6"], tab["rface"]),
                                 e.set_cooling_tables(tab["cool_omega"], tab["cool_temp"]))


def _disk_engine(n, prec):
    desc = pnbbh.pnbbh_desc(n, precision=PREC[prec])
    tab = pnbbh.pnbbh_tables(desc)
    metric = pnbbh.pnbbh_coords(spacetime=hg.DYN_PN_BINARY)
    return desc, tab, metric, lambda e: (e.set_dynamic_metric(metric), e.set_cell_data(tab["cell6"], tab["rface"]),
                                         e.set_cooling_tables(*pnbbh.pn_cooling_tables(tab)))


def prepare(case, seed):
    kind, prec = case["kind"], case["prec"]
    if kind == "batch":
        grids = [_minkowski_grid(k, n, prec, s) for k, n, s in _members(case, seed)]
        batch = hg.Batch(0, case["members"])
        for g in grids:
            g.load()
            batch.add(g.engine)
        return dict(case=case, grids=grids, batch=batch)
    n = (case["n1"], case["n2"], case["n3"])
    if kind in ("tube", "loop", "wave"):
        return dict(case=case, grid=_minkowski_grid(kind, n, prec, seed))
    # torus and disk: the setup's initial data, taken by the FP64 form past
    # the ramp of the first time step (each step may grow by 1.3 from 1e-5)
    if kind == "torus":
        desc, tab, tables = _torus_engine(n, "fp64")
        e = hg.Engine(desc)
        tables(e)
        torus.set_torus(e, desc, tab, seed=seed, return_prims=False)
    else:
        desc, tab, metric, tables = _disk_engine(n, "fp64")
        e = hg.Engine(desc)
        tables(e)
        pnbbh.set_disk(e, desc, tab, metric, seed=seed, return_prims=False)
    e.set_time(0.0, desc.dx[0])
    t, dt = e.step(40)
    p = e.download()
    e.close()
    desc.precision = PREC[prec]
    g = Grid(desc, p, t, dt)
    tables(g.engine)
    return dict(case=case, grid=g)


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        for g in state["grids"]:
            g.load()
        for _ in range(case["steps"]):
            t, dt = state["batch"].step()
        return dict(p=[g.engine.download(g.out) for g in state["grids"]], t=t, dt=dt)
    g = state["grid"]
    g.load()
    t, dt = g.engine.step(case["steps"])
    out = dict(p=g.engine.download(g.out), t=t, dt=dt)
    if case["prec"] == "fp64":
        out["fails"] = g.engine.fail_counts().astype(np.int64)
    return out


def _zones(case):
    if case["kind"] == "batch":
        return sum(n[0] * n[1] * n[2] for _, n, _ in _members(case, 0))
    return case["n1"] * case["n2"] * case["n3"]


def work(case):
    """Per zone and substep: the eight primitives read and written once, the
    floors read; faces 800 operations for each resolved direction (two states,
    their speeds and eight components), the reconstruction 200 of them, 800
    for the conserved update, the EMFs and the inversion, 400 more in a curved
    metric; the time-dependent metric is 86 doubles a zone and level.  The
    transfers move the primitives once each way."""
    z = _zones(case) * case["steps"] * 2
    dims = 3 if case["kind"] == "batch" else sum(case[k] > 1 for k in ("n1", "n2", "n3"))
    per = 800 * dims + 800 + (400 if case["kind"] in ("torus", "disk") else 0)
    b = 144 * z + 128 * _zones(case)
    if case["kind"] == "disk":
        b, per = b + 8 * 86 * z, per + 1500
    return {"bytes": b, "flops": per * z}


def tolerance(case):
    """fp64: the form's own contract.  The others: about four times the
    distance of the three forms from one another over a pass."""
    if case["prec"] == "fp64":
        return "exact"
    if case["prec"] == "fma":  # rounding of 64 bits, through the inversions and the entropy fix
        return {"rel": 1e-12, "max": 1e-8}
    if case["kind"] == "torus":  # FP32 face fluxes, whose differences are small against them
        return {"rel": 1e-5, "max": 2e-2}
    return {"rel": 3e-7, "max": 1e-5}


# --------------------------------------------------------------------------
# exact(): the steps of a Minkowski grid in plain torch at 64 bits

RHO, UU, U1, U2, U3, B1, B2, B3 = range(8)


class Plain:
    """PPM_MC or MC reconstruction, HLL fluxes, parabolic flux-CT, two-stage
    stepping and the two-dimensional Newton inversion on a Cartesian grid in
    flat space.  Arrays hold every ghost zone; a direction of one zone holds
    that zone once and has no fluxes to difference."""

    def __init__(self, desc, p, t, dt):
        n = (desc.n1, desc.n2, desc.n3)
        self.n, self.gam, self.cour = n, desc.gam, desc.cour
        self.dx = [desc.dx[a + 1] for a in range(3)]
        self.ppm, self.wrap = desc.recon_type == hg.RECON_PPM_MC, desc.bc_type == hg.BC_CARTESIAN_PERIODIC
        self.t, self.dt = t, dt
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        p = p[tuple(slice(None) if m > 1 else slice(NG, NG + 1) for m in n)]
        self.p = torch.from_numpy(np.ascontiguousarray(np.moveaxis(p, -1, 0))).to(dev)
        self.phys = tuple(slice(NG, NG + m) if m > 1 else slice(0, 1) for m in n)

    def at(self, x, a, m):
        """x of the zone m further along direction a."""
        return x if self.n[a] == 1 else torch.roll(x, -m, dims=x.dim() - 3 + a)

    @staticmethod
    def mc(a, b):
        r = 0.5 * (a + b)
        r = torch.where(3 * b.abs() <= a.abs(), 2 * b, r)
        r = torch.where(3 * a.abs() <= b.abs(), 2 * a, r)
        return torch.where(a * b <= 0, torch.zeros_like(r), r)

    def edges(self, y, a, ppm=True):
        """Left and right edge values of every zone along direction a."""
        if self.n[a] == 1:
            return y, y
        d = self.at(y, a, 1) - y
        q = self.mc(self.at(d, a, -1), d)
        if not ppm:
            return y - 0.5 * q, y + 0.5 * q
        r = 0.5 * (self.at(y, a, 1) + y) - (self.at(q, a, 1) - q) / 6
        l = self.at(r, a, -1)
        up = r > l
        lo, hi = 3 * y - 2 * r, 3 * y - 2 * l
        ln = torch.where(torch.where(up, 3 * y > l + 2 * r, 3 * y < l + 2 * r), lo, l)
        rn = torch.where(torch.where(up, 3 * y < 2 * l + r, 3 * y > 2 * l + r), hi, r)
        flat = (r - y) * (y - l) <= 0
        return torch.where(flat, y, ln), torch.where(flat, y, rn)

    def state(self, p):
        v, B = p[U1:B1], p[B1:]
        ut = torch.sqrt(1 + (v * v).sum(0))
        bt = (B * v).sum(0)
        b = (B + bt * v) / ut
        bsq = (b * b).sum(0) - bt * bt
        pg = (self.gam - 1) * p[UU]
        return dict(ut=ut, v=v, bt=bt, b=b, bsq=bsq, pg=pg, eta=p[RHO] + p[UU] + pg + bsq, ptot=pg + 0.5 * bsq)

    def flux(self, p, s, a):
        """Conserved variables (a None) or fluxes along direction a."""
        u, b = (s["ut"], s["bt"]) if a is None else (s["v"][a], s["b"][a])
        f = torch.empty_like(p)
        f[RHO] = p[RHO] * u
        f[UU] = -s["eta"] * u * s["ut"] + b * s["bt"] + f[RHO]
        f[U1:B1] = s["eta"] * u * s["v"] - b * s["b"]
        f[B1:] = s["b"] * u - b * s["v"]
        if a is None:
            f[UU] += s["ptot"]
        else:
            f[U1 + a] += s["ptot"]
        return f

    def speeds(self, p, s, a):
        c = ((self.gam * s["pg"] + s["bsq"]) / s["eta"]).clamp(0, 1)
        u, ut = s["v"][a], s["ut"]
        A = ut * ut - (ut * ut - 1) * c
        B = u * ut - u * ut * c
        C = u * u - (u * u + 1) * c
        d = torch.sqrt((B * B - A * C).clamp(min=0))
        return (B + d) / A, (B - d) / A

    def hll(self, p, a):
        """HLL fluxes at the lower face of every zone, and the largest speed over the physical faces."""
        l, r = self.edges(p, a, self.ppm)
        pl, pr = self.at(r, a, -1), l
        sl, sr = self.state(pl), self.state(pr)
        (xl, nl), (xr, nr) = self.speeds(pl, sl, a), self.speeds(pr, sr, a)
        cp = torch.maximum(xl, xr).clamp(min=0)
        cm = torch.maximum(-nl, -nr).clamp(min=0)
        F = (cp * self.flux(pl, sl, a) + cm * self.flux(pr, sr, a)
             - cp * cm * (self.flux(pr, sr, None) - self.flux(pl, sl, None))) / (cp + cm + 1e-15)
        return F, float(torch.maximum(cp, cm)[self.phys].max())

    def emf(self, F, G, a, b):
        """Corner EMF from F along direction b and G along direction a."""
        fl, fr = self.edges(F, b)
        gl, gr = self.edges(G, a)
        return self.at(fr, b, -1) + fl - self.at(gr, a, -1) - gl

    def update(self, p0, p, dt):
        """Conserved variables a time dt after those of p0, with the fluxes of p."""
        F, c = zip(*(self.hll(p, a) for a in range(3)))
        E = (self.emf(F[1][B3], F[2][B2], 1, 2), self.emf(F[2][B1], F[0][B3], 2, 0), self.emf(F[0][B2], F[1][B1], 0, 1))
        U = self.flux(p0, self.state(p0), None)
        for a in range(3):
            if self.n[a] > 1:
                U[:B1] -= dt / self.dx[a] * (self.at(F[a], a, 1) - F[a])[:B1]
        for i in range(3):  # curl of the corner EMFs, averaged to the faces
            j, k = (i + 1) % 3, (i + 2) % 3
            for a, e, sign in ((j, k, -1.0), (k, j, 1.0)):
                if self.n[a] > 1:
                    x = E[e] + self.at(E[e], i, 1)
                    U[B1 + i] -= sign * 0.125 * dt / self.dx[a] * (self.at(x, a, 1) - x)
        return U, c

    def invert(self, U, p):
        """Primitives of U: Newton in W = w gamma^2 and v^2 from the guess p."""
        g = (self.gam - 1) / self.gam
        D, B = U[RHO], U[B1:]
        Q0, Q = U[UU] - U[RHO], U[U1:B1]
        Bsq, QB = (B * B).sum(0), (Q * B).sum(0)
        QBsq, Qsq, Qn = QB * QB, (Q * Q).sum(0), Q0
        gsq = 1 + (p[U1:B1] ** 2).sum(0)
        W = (D / torch.sqrt(gsq) + self.gam * p[UU]) * gsq
        v = ((W * W * Qsq + QBsq * (Bsq + 2 * W)) / (W * W * (Bsq + W) ** 2)).clamp(max=1 - 1e-15)
        for _ in range(12):  # quadratic: the guess is the state a step before
            s = torch.sqrt(1 - v)
            dPv = g * (0.5 * D / s - W)
            t3 = Bsq + W
            t16 = QBsq / (W * W)
            t11 = Qsq - v * t3 * t3 + t16 * (Bsq + 2 * W)
            t18 = -Qn - 0.5 * Bsq * (1 + v) + 0.5 * t16 - W + g * (W * (1 - v) - D * s)
            t24 = t16 / W
            t25 = -1 + g * (1 - v) - t24
            t21 = 1 / (t3 * (t25 * t3 + (Bsq - 2 * dPv) * (t16 + v * W) / W))
            dW = -((dPv - 0.5 * Bsq) * t11 + t3 * t3 * t18) * t21
            dv = -(-t25 * t11 - 2 * (v + t24) * t3 * t18) * t21
            W, v = (W + dW).abs(), (v + dv).clamp(0, 1 - 1e-15)
        s = torch.sqrt(1 - v)
        out = torch.empty_like(U)
        out[RHO] = D * s
        out[UU] = (W * (1 - v) - out[RHO]) / self.gam
        out[U1:B1] = (Q + QB / W * B) / (s * (W + Bsq))
        out[B1:] = B
        return out

    def bounded(self, p):
        for a, m in enumerate(self.n):
            if m > 1:
                x = torch.arange(m + 2 * NG, device=p.device) - NG
                p = p.index_select(a + 1, NG + (x % m if self.wrap else x.clamp(0, m - 1)))
        return p

    def step(self):
        p0 = self.p
        U, _ = self.update(p0, p0, 0.5 * self.dt)
        half = self.bounded(self.invert(U, p0))
        U, c = self.update(p0, half, self.dt)
        self.p = self.bounded(self.invert(U, p0))
        self.t += self.dt
        new = self.cour * math.sqrt((1 / 3) / sum((x / d) ** 2 for x, d in zip(c, self.dx)))
        self.dt = min(new, 1.3 * self.dt)

    def whole(self):
        p = np.moveaxis(self.p.cpu().numpy(), 0, -1)
        for a, m in enumerate(self.n):
            if m == 1:
                p = np.repeat(p, 1 + 2 * NG, axis=a)
        return np.ascontiguousarray(p)


def _plain(kind, n, seed, steps):
    prob, p, dt = _minkowski(kind, n, hg.PREC_FP64, seed)
    s = Plain(prob.desc, p, 0.0, dt)
    for _ in range(steps):
        s.step()
    return s


def exact(case, seed):
    if case["kind"] in ("torus", "disk") or _zones(case) * case["steps"] > 1e8:
        # the entropy fix's tree in plain torch, or the largest grid: over 20 s
        return None
    if case["kind"] == "batch":
        m = [_plain(k, n, s, case["steps"]) for k, n, s in _members(case, seed)]
        return dict(p=[s.whole() for s in m], t=np.array([s.t for s in m]), dt=np.array([s.dt for s in m]))
    s = _plain(case["kind"], (case["n1"], case["n2"], case["n3"]), seed, case["steps"])
    return dict(p=s.whole(), t=s.t, dt=s.dt)
