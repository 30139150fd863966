"""Cases of work that users of this library have it do, for timing it.

Each case is one call sequence of a user's program through the public
Python interface: runs of the 3D and 2D particle-mesh step from records in
host memory (load, assign the mass, step, unload), runs with time-step
zones, the forces and potentials of a given set of particles, the
smooth-field-particle (SFP) sum and time loop, a batched ensemble, and the
gradient of a run.  Sizes come from bench.py's workloads, the tests'
configurations (the reference's own run100 and run200 among them) and the
ranges around them.

``listed`` gives the cases, ``draw`` one more of the same ranges,
``prepare`` what the program holds before the call, ``run`` one pass,
``work`` the bytes and operations the pass cannot do without, ``exact`` the
same results in FP64 from plain torch.
"""
import json
import math
import os

import numpy as np
import torch
import torch.utils.checkpoint

BASIS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden", "aj07.json")

# the most work any case may ask for, in particle-steps of a 3D run
COST_MAX = 10_000_000 * 60


# ---------------------------------------------------------------------------
# the cases
def grid3(nr=128, na=256, ngz=125, ng=17, map="log"):
    return dict(ndim=3, nr=nr, na=na, ngz=ngz, ng=ng, map=map)


def grid2(nr=64, na=128, ng=9, map="log"):
    return dict(ndim=2, nr=nr, na=na, ngz=1, ng=ng, map=map)


def listed():
    return [
        # the 3D workload the framework is benchmarked on: a disc of 10M
        # particles between two dumps of its particles
        dict(name="p3d-10M", kind="run", **grid3(), n=10_000_000, steps=60),
        # the same grid with fewer particles, where the field solve counts as
        # much as the particles; two-float positions, as long runs use
        dict(name="p3d-1M-compensated", kind="run", **grid3(), n=1_000_000, steps=60, comp=True),
        # a grid of ragged sizes on the reference's default radial map, with a
        # halo: an ordinary run of the p3d example's size
        dict(name="p3d-ragged-200k", kind="run", **grid3(85, 126, 75, 9, "std"), n=203_117, steps=60, halo=1,
             spline=True),
        # the 27-point quadratic scheme (the 'inte 3' card)
        dict(name="p3d-quadratic-500k", kind="run", **grid3(64, 128, 45, 17), n=500_000, steps=40, quad=True),
        # the size of the reference's p2d examples: latency and launches
        dict(name="p2d-100k", kind="run", **grid2(), n=100_000, steps=200),
        # a large 2D run in a halo
        dict(name="p2d-3M", kind="run", **grid2(128, 256, 9), n=3_000_000, steps=100, halo=1),
        # the reference's run100: two time-step zones, two sectors, a fixed
        # axisymmetric force in place of m = 0
        dict(name="p2d-zones-15k", kind="zones", **grid2(93, 128, 3, "std"), n=15_000, steps=100, nsect=2, halo=2,
             nzones=2),
        # forces and potentials at given positions (an analysis program)
        dict(name="p3d-forces-1M", kind="forces", **grid3(), n=1_000_000),
        # the SFP coefficient sum of a loaded set of particles
        dict(name="sfp-sum-20M", kind="sfp_sum", n=20_000_000, maxm=8, maxn=19, precision=0),
        # a run in the SFP field
        dict(name="sfp-run-1M", kind="sfp_run", n=1_000_000, maxm=8, maxn=19, steps=60, precision=0),
        # a parameter study: independent discs advanced together
        dict(name="ensemble-16", kind="ensemble", **grid2(), discs=16, nmin=20_000, nmax=400_000, steps=256),
        # the gradient of the bar amplitude with respect to the initial state
        dict(name="adjoint-400k", kind="adjoint", **grid2(128, 256, 9), n=400_000, steps=100, ckpt=25, halo=1),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _grid3_draw(rng):
    ngz = rng.choice([15, 25, 27, 45, 75, 81, 125])
    g = grid3(rng.randint(40, 128), 2 * rng.randint(24, 128), ngz, rng.randint(3, 17))
    if rng.random() < 0.4:
        g["nr"] -= g["nr"] % 4
    if rng.random() < 0.3:
        # the default map's edge, e^(2 pi (nr - 1) / na) - 1: the p3d example's shape
        g.update(map="std", na=2 * (3 * g["nr"] // 4))
    return g


def _grid2_draw(rng):
    g = grid2(rng.randint(40, 140), 2 * rng.randint(24, 128), rng.randint(2, 17))
    if rng.random() < 0.3:
        g.update(map="std", na=2 * (3 * g["nr"] // 4))
    return g


def draw(rng):
    kind = rng.choice(["run3", "run3", "run3", "run2", "run2", "zones", "forces", "sfp_sum", "sfp_run", "ensemble",
                       "adjoint"])
    halo = rng.choice([0, 0, 1])
    if kind == "run3":
        c = dict(kind="run", **_grid3_draw(rng), n=int(_log(rng, 20_000, 6_000_000)), steps=rng.randint(20, 60), halo=halo)
        r = rng.random()
        if r < 0.2:
            c.update(quad=True, n=min(c["n"], 1_500_000))
        elif r < 0.4:
            c.update(comp=True)
        if rng.random() < 0.25:
            c.update(spline=True)
    elif kind == "run2":
        c = dict(kind="run", **_grid2_draw(rng), n=int(_log(rng, 5_000, 4_000_000)), steps=rng.randint(50, 200), halo=halo,
                 comp=rng.random() < 0.25)
    elif kind == "zones":
        three = rng.random() < 0.4
        g = grid3(64, 96, 45, 9, "std") if three else grid2(93, 128, 3, "std")
        c = dict(kind="zones", **g, n=int(_log(rng, 10_000, 300_000)), steps=4 * rng.randint(10, 25),
                 nsect=1 if three else 2, halo=1 if three else 2, nzones=rng.choice([2, 3]))
    elif kind == "forces":
        c = dict(kind="forces", **(_grid3_draw(rng) if rng.random() < 0.6 else _grid2_draw(rng)),
                 n=int(_log(rng, 10_000, 3_000_000)), halo=halo)
    elif kind == "sfp_sum":
        c = dict(kind="sfp_sum", n=int(_log(rng, 100_000, 20_000_000)), maxm=rng.randint(2, 8), maxn=rng.randint(5, 19),
                 precision=rng.choice([0, 0, 2]))
    elif kind == "sfp_run":
        c = dict(kind="sfp_run", n=int(_log(rng, 50_000, 3_000_000)), maxm=rng.randint(2, 8), maxn=rng.randint(5, 19),
                 steps=rng.randint(20, 60), precision=rng.choice([0, 0, 2]))
    elif kind == "ensemble":
        nmin = int(_log(rng, 5_000, 30_000))
        c = dict(kind="ensemble", **grid2(rng.randint(40, 72), 2 * rng.randint(32, 72), rng.randint(3, 9)),
                 discs=rng.randint(4, 32), nmin=nmin, nmax=nmin * rng.randint(2, 12), steps=rng.randint(64, 256))
    else:
        c = dict(kind="adjoint", **grid2(rng.randint(48, 128), 2 * rng.randint(32, 128), rng.randint(3, 9)),
                 n=int(_log(rng, 10_000, 500_000)), steps=rng.randint(20, 100), ckpt=rng.randint(5, 50), halo=halo)
    if "steps" in c and c["kind"] == "run" and c["n"] * c["steps"] > COST_MAX:
        c["steps"] = max(1, COST_MAX // c["n"])
    return c


# ---------------------------------------------------------------------------
# grids and discs
def _params(c):
    """Grid and run parameters in grid units: the log map spans r = 0.05 .. 5
    at one grid unit per disc scale; the default map takes the disc's scale as
    a sixth of 0.9 of its edge's radius per length unit."""
    p = dict(halo=c.get("halo", 0), nsect=c.get("nsect", 1), skip=(0,) if c.get("halo") == 2 else ())
    dt = 0.02 if c["ndim"] == 3 else 0.025
    if c["map"] == "log":
        p.update(rmap=1, a=math.log(100.0) / (c["nr"] - 1), r0=0.05, lscale=1.0, rmax=4.8, softl=0.1 if c["nr"] >= 60 else 0.2)
        dz = {15: 0.1, 25: 0.08, 27: 0.08}.get(c["ngz"], 0.04)
    else:
        edge = math.exp(2 * math.pi * (c["nr"] - 1) / c["na"]) - 1
        p.update(rmap=0, a=0.0, r0=0.0, lscale=edge / 6.0, rmax=5.0)
        last = edge - (math.exp(2 * math.pi * (c["nr"] - 2) / c["na"]) - 1)
        p["softl"] = max(0.1 * p["lscale"], last / 4)
        dz = 0.5 * p["softl"]
    p["dzg"] = dz if c["ndim"] == 3 else 0.0
    L = p["lscale"]
    p["dt"], p["z0"] = dt, 0.1
    p["halo_rc"] = {0: 1.0, 1: L, 2: 1.1 * L}[p["halo"]]
    p["halo_v2"] = {0: 0.0, 1: 0.49 * L * L * dt * dt, 2: L ** 3 * dt * dt}[p["halo"]]
    return p


def _config(c, pmass):
    import galaxy_b200 as gb
    p = _params(c)
    flags = (gb.GX_FLAG_COMPENSATED if c.get("comp") else 0) | (gb.GX_FLAG_QUADRATIC if c.get("quad") else 0)
    return gb.make_config(c["ndim"], c["nr"], c["na"], ngz=c["ngz"], dzg=p["dzg"], ng=c["ng"], nsect=p["nsect"],
                          skip=p["skip"], rmap=p["rmap"], rmap_a=p["a"], rmap_r0=p["r0"], softl=p["softl"],
                          tsoft=2 if c.get("spline") else 1, pmass=pmass, halo=p["halo"], halo_v2=p["halo_v2"],
                          halo_rc=p["halo_rc"], flags=flags)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _disc(c, n, seed):
    """A Kuzmin-Toomre disc as galaxy_b200/disk.py makes it (Q = 1.2, sech^2
    layer), on the GPU: records [n, 2 ndim] in grid units and the particle mass."""
    p, g = _params(c), _gen(seed)
    dev, f8 = "cuda", torch.float64
    def u(): return torch.rand(n, generator=g, device=dev, dtype=f8)
    def z(): return torch.randn(n, generator=g, device=dev, dtype=f8)
    r = (1 / (1 - u() * (1 - (1 + p["rmax"] ** 2) ** -0.5)) ** 2 - 1).sqrt()
    phi = 2 * math.pi * u()
    v2 = 0.49 if p["halo"] == 1 else 0.0
    vc2 = r * r / (1 + r * r) ** 1.5 + v2 * r * r / (r * r + 1)
    om2 = vc2 / (r * r).clamp_min(1e-12)
    kap2 = (r * (-3 * r / (1 + r * r) ** 2.5 - 2 * v2 * r / (r * r + 1) ** 2) + 4 * om2).clamp_min(1e-12)
    sig = (1 + r * r) ** -1.5 / (2 * math.pi)
    sr = 3.36 * 1.2 * sig / kap2.sqrt()
    vr, vp = z() * sr, vc2.sqrt() + z() * sr * (kap2 / (4 * om2)).sqrt()
    cs, sn = phi.cos(), phi.sin()
    x = [r * cs, r * sn]
    v = [vr * cs - vp * sn, vr * sn + vp * cs]
    if c["ndim"] == 3:
        x.append(p["z0"] * torch.atanh((2 * u() - 1).clamp(-1 + 1e-12, 1 - 1e-12)))
        v.append(z() * (math.pi * sig * p["z0"]).sqrt())
    L, dt = p["lscale"], p["dt"]
    rec = torch.stack([q * L for q in x] + [q * (L * dt) for q in v], 1).float()
    return rec, L ** 3 * dt * dt / n


def _zones(c):
    """Step factors and radii of the zones (run100: 1, 2; run200: 1, 2, 4)."""
    L = _params(c)["lscale"]
    return ([1, 2], [0.0, 3.0 * L]) if c["nzones"] == 2 else ([1, 2, 4], [0.0, L, 2.5 * L])


def _exp_disc(n, seed):
    """An exponential disc truncated at r = 6 on near-circular orbits: records
    (x, y, vx, vy), as the SFP configuration of bench.py draws its positions."""
    g = _gen(seed)
    rr = torch.linspace(0, 6, 100001, device="cuda", dtype=torch.float64)
    cdf = 1 - (1 + rr) * torch.exp(-rr)
    cdf = cdf / cdf[-1].clone()
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    k = torch.searchsorted(cdf, u).clamp(1, rr.numel() - 1)
    r = rr[k - 1] + (u - cdf[k - 1]) / (cdf[k] - cdf[k - 1]) * (rr[k] - rr[k - 1])
    phi = 2 * math.pi * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    vc = (r * r / (1 + r * r) ** 1.5).sqrt()
    return torch.stack([r * phi.cos(), r * phi.sin(), -vc * phi.sin(), vc * phi.cos()], 1).float()


def _counts(c):
    rng = np.random.default_rng(12345)
    return np.round(np.exp(rng.uniform(math.log(c["nmin"]), math.log(c["nmax"]), c["discs"]))).astype(int)


class State(dict):
    """What the program holds; the library's handles are closed with it."""

    def __del__(self):
        try:
            self["handle"].close()
        except Exception:
            pass


class Kept(np.ndarray):
    """The contents of a page-locked buffer, which lives as long as they do."""


def _out(shape):
    from galaxy_b200 import PinnedArray
    a = PinnedArray(shape)
    v = a.array.view(Kept)
    v.owner = a
    return v


def _pinned(rec):
    from galaxy_b200 import PinnedArray
    a = PinnedArray(tuple(rec.shape))
    a.array[...] = rec.cpu().numpy()
    return a


def prepare(case, seed):
    from galaxy_b200 import Galaxy
    c = case
    if c["kind"].startswith("sfp"):
        from galaxy_b200.sfp import Basis, Sfp
        rec = _pinned(_exp_disc(c["n"], seed))
        h = Sfp(Basis.from_json(BASIS, maxm=c["maxm"], maxn=c["maxn"]), 6.0)
        h.load(rec.array)
        return State(case=c, handle=h, rec=rec)
    if c["kind"] == "ensemble":
        # a study in progress: the discs are loaded, and every pass advances them
        from galaxy_b200.ensemble import Ensemble
        recs, pms = zip(*(_disc(c, int(n), seed * 1000 + d) for d, n in enumerate(_counts(c))))
        h = Ensemble(_config(c, 1.0), [r.cpu().numpy() for r in recs], np.array(pms, np.float32), max_steps=500_000)
        h.tune()
        return State(case=c, handle=h)
    rec, pm = _disc(c, c["n"], seed)
    rec = _pinned(rec)
    h = Galaxy(_config(c, pm))
    h.greenm()
    if c["kind"] == "zones":
        h.set_zones(*_zones(c))
    return State(case=c, handle=h, rec=rec, out=_out(rec.array.shape))


def run(state):
    c, h = state["case"], state["handle"]
    if c["kind"] == "sfp_sum":
        return {"coeff": h.sum(1.0 / c["n"], c["precision"])}
    if c["kind"] == "sfp_run":
        h.load(state["rec"].array)
        coeff = h.step(c["steps"], 0.01, 1.0 / c["n"], c["precision"])
        return {"coeff": coeff, "particles": h.unload()}
    if c["kind"] == "ensemble":
        h.step(c["steps"])
        return {"particles": h.unload()}
    h.loadup_ptr(state["rec"].ptr, c["n"])
    h.masset()
    if c["kind"] == "forces":
        h.findf(True)
        acc, pot = h.getacc()
        return {"acc": acc, "pot": pot}
    if c["kind"] == "adjoint":
        # the drift it also reports measures rounding alone
        J, grad, dth, _ = h.adjoint(c["steps"], c["ckpt"])
        return {"J": J, "grad": grad, "dtheta": dth}
    h.step(c["steps"])
    h.unload_ptr(state["out"].owner.ptr)
    return {"particles": state["out"]}


def work(case):
    """One step reads and writes every particle's phase space, reads the Green
    table of the force components once, and writes and reads the mass and the
    force grids; per particle it interpolates and assigns with 2^ndim (27:
    quadratic) weights per component."""
    c = case
    if c["kind"].startswith("sfp"):
        deg = 32
        steps = c.get("steps", 0)
        f = 2.0 * c["n"] * deg * (2 * c["maxm"] + 1)  # moments of the Chebyshev terms and harmonics
        if not steps:
            return dict(bytes=8.0 * c["n"], flops=f)
        return dict(bytes=c["n"] * (32.0 * steps + 8 + 32), flops=(steps + 1) * f + steps * 40.0 * c["n"] * (c["maxm"] + 1))
    nd, mesh = c["ndim"], c["nr"] * c["na"] * c["ngz"]
    nw = 27 if c.get("quad") else 2 ** nd
    nkz = c["ngz"] + 1 if nd == 3 else 1
    act = [m for m in range(c["ng"]) if m % c.get("nsect", 1) == 0 and not (m == 0 and c.get("halo") == 2)]
    green = nd * len(act) * nkz * c["nr"] ** 2
    grids = 4.0 * mesh * (2 + 2 * nd)
    if c["kind"] == "ensemble":
        n = float(sum(_counts(c)))
        per = dict(bytes=n * 32 + c["discs"] * grids + 4 * green, flops=n * nw * (2 * nd + 4) + c["discs"] * 4.0 * green)
        return dict(bytes=c["steps"] * per["bytes"] + 16 * n, flops=c["steps"] * per["flops"])
    n = float(c["n"])
    step = dict(bytes=n * 16 * nd + 4.0 * green + grids, flops=n * nw * (2 * nd + 4) + 8.0 * green)
    host = n * 16 * nd
    if c["kind"] == "forces":
        return dict(bytes=n * 8 * nd + n * 4 * (nd + 1) + 4.0 * green * (nd + 1) / nd + grids, flops=step["flops"])
    if c["kind"] == "adjoint":
        # forward: a step; backward: the state and the gradient read and written, both solves
        return dict(bytes=c["steps"] * (3 * step["bytes"] + n * 32) + n * 32, flops=c["steps"] * 3.5 * step["flops"])
    return dict(bytes=c["steps"] * step["bytes"] + host, flops=c["steps"] * step["flops"])


# ---------------------------------------------------------------------------
# the same results in FP64 from torch alone
class Mesh:
    """The particle-mesh method on the polar grid: cloud-in-cell (or
    quadratic) weights, the softened kernel sampled on the grid, convolution
    over spokes (filtered to the active harmonics) and planes by FFT and over
    rings directly."""

    def __init__(self, c, pmass, pot=False):
        p = _params(c)
        f = lambda v: float(np.float32(v))  # noqa: E731  the configuration holds FP32 values
        self.c, self.pm = c, f(pmass)
        self.nd, self.nr, self.na, self.ngz = c["ndim"], c["nr"], c["na"], c["ngz"]
        self.quad = bool(c.get("quad"))
        self.a = f(p["a"]) if p["a"] > 0 else 2 * math.pi / self.na
        self.log = p["rmap"] == 1
        self.off = -math.log(f(p["r0"])) / self.a if self.log else 0.0
        self.dz = f(p["dzg"])
        self.zm = 0.5 * self.dz * (self.ngz - 1)
        self.rin = math.exp(-self.a * self.off) if self.log else 0.0
        self.rout = float(self.grofu(torch.tensor(float(self.nr - 1))))
        self.halo = p["halo"]
        self.v2 = torch.tensor(f(p["halo_v2"]), dtype=torch.float64, device="cuda")
        self.rc = torch.tensor(f(p["halo_rc"]), dtype=torch.float64, device="cuda")
        self.m = [m for m in range(min(c["ng"], self.na // 2 + 1)) if m % p["nsect"] == 0 and m not in p["skip"]]
        self.K = self.kernels(f(p["softl"]), bool(c.get("spline")), pot)
        th = 2 * math.pi * torch.arange(self.na, device="cuda", dtype=torch.float64) / self.na
        self.cos, self.sin = th.cos(), th.sin()

    def grofu(self, u):
        return torch.exp(self.a * (u - self.off)) - (0.0 if self.log else 1.0)

    def kernels(self, eps, spline, pot):
        nr, na, nz = self.nr, self.na, self.ngz
        r = self.grofu(torch.arange(nr, device="cuda", dtype=torch.float64))
        th = 2 * math.pi * torch.arange(na, device="cuda", dtype=torch.float64) / na
        nsep = nz + 1 if self.nd == 3 else 1
        z = (self.dz * torch.arange(nsep, device="cuda", dtype=torch.float64)).view(1, 1, -1, 1)
        ct, st = th.cos().view(1, 1, 1, -1), th.sin().view(1, 1, 1, -1)
        rf = r.view(1, nr, 1, 1)
        types = ["r", "t"] + (["z"] if self.nd == 3 else []) + (["p"] if pot else [])
        nk = 2 * nz if self.nd == 3 else 1
        out = {t: torch.zeros(len(self.m), nk, nr, nr, dtype=torch.complex128, device="cuda") for t in types}
        block = max(1, int(6e7 / (nr * nsep * na)))
        for i0 in range(0, nr, block):
            rs = r[i0:i0 + block].view(-1, 1, 1, 1)
            d2 = rs * rs + rf * rf - 2 * rs * rf * ct + z * z
            if spline:
                d = d2.clamp_min(0).sqrt()
                s = d / eps
                m = torch.where(s < 1, 4 * s ** 3 * (0.333333333 - 0.3 * s * s + 0.125 * s ** 3),
                                torch.where(s < 2, -1 / 15 + s ** 3 * (2.6666667 - 3 * s + 1.2 * s * s - 0.166666667 * s ** 3),
                                            torch.ones_like(s)))
                w = torch.where(d2 > 0, m / d.clamp_min(1e-300) ** 3, torch.zeros_like(m))
                x = s
                ph = torch.where(x < 1, -1.4 + x * x * (0.6666667 - 0.3 * x * x + 0.1 * x ** 3),
                                 torch.where(x < 2, -1.6 + 1 / (15 * x.clamp_min(1e-9)) +
                                             x * x * (1.33333333 - x + 0.3 * x * x - 0.033333333 * x ** 3),
                                             -1 / x.clamp_min(1e-9))) / eps if pot else None
            else:
                w = (d2 + eps * eps) ** -1.5
                ph = -(d2 + eps * eps) ** -0.5 if pot else None
            for t in types:
                k = {"r": lambda: (rs * ct - rf) * w, "t": lambda: -rs * st * w, "z": lambda: -z * w, "p": lambda: ph}[t]()
                k = torch.fft.rfft(k, dim=3)[..., self.m]                  # [is, ir, sep, m]
                if t == "t" and self.m[-1] == na // 2:
                    k[..., -1] = 0
                if self.nd == 3:
                    inner = k[:, :, 1:nz].flip(2)
                    if t == "z":
                        k[:, :, nz] = 0
                        inner = -inner
                    k = torch.fft.fft(torch.cat([k, inner], 2), dim=2)     # the doubled grid
                out[t][..., i0:i0 + rs.shape[0]] = k.permute(3, 2, 1, 0)    # [m, kz, ir, is]
        return out

    def cells(self, x):
        """Corner cells [n, corners] and their weights; zero weights off the grid."""
        nr, na, nz = self.nr, self.na, self.ngz
        with torch.no_grad():
            rr = x[:, :2].square().sum(1).sqrt()
            on = (rr <= self.rout) & (rr >= self.rin)
            if self.nd == 3:
                on = on & (x[:, 2].abs() <= self.zm)
        safe = torch.where(on, torch.ones_like(rr), torch.zeros_like(rr))
        px = torch.where(on, x[:, 0], torch.ones_like(rr))
        py = torch.where(on, x[:, 1], torch.zeros_like(rr))
        r = (px * px + py * py).sqrt() if not self.log else None
        u = (0.5 * torch.log(px * px + py * py) / self.a + self.off) if self.log else torch.log1p(r) / self.a
        t = torch.atan2(py, px) * (na / (2 * math.pi))
        t = torch.where(t < 0, t + na, t)
        zz = torch.where(on, (x[:, 2] + self.zm) / self.dz, torch.zeros_like(rr)) if self.nd == 3 else None
        with torch.no_grad():
            h = 0.5 if self.quad else 0.0
            ju = (u + h).floor().clamp(1 if self.quad else 0, nr - 2)
            jt = (t + h).floor()
            jz = (zz + h).floor().clamp(0, nz - 2) if self.nd == 3 else None
        def lin(d): return [1 - d, d]
        def quad(d): return [0.5 - d + 0.5 * d * d, 0.5 + d - d * d, 0.5 * d * d]
        fw = (lambda q, j: quad(q + 0.5 - j)) if self.quad else (lambda q, j: lin(q - j))
        lo = -1 if self.quad else 0
        ft, fu = fw(t, jt), fw(u, ju)
        fz = fw(zz, jz) if self.nd == 3 else [torch.ones_like(u)]
        idx, wt = [], []
        for k, a in enumerate(fu):
            for j, b in enumerate(fz):
                for i, e in enumerate(ft):
                    it = (jt + (i + lo)) % na
                    iz = jz + (j + lo) if self.nd == 3 else 0
                    ix = ((ju + (k + lo)) * nz + iz) * na + it
                    idx.append(ix.clamp(0, nr * nz * na - 1).long())
                    wt.append(a * b * e * safe)
        return on, torch.stack(idx, 1), torch.stack(wt, 1)

    def mass(self, cell):
        _, idx, wt = cell
        m = torch.zeros(self.nr * self.ngz * self.na, dtype=torch.float64, device="cuda")
        for k in range(idx.shape[1]):
            m = m.index_add(0, idx[:, k], wt[:, k])
        return m

    def field(self, mass):
        """(fx, fy[, fz][, potential]) [mesh, components] of an unscaled mass array."""
        nr, na, nz = self.nr, self.na, self.ngz
        s = torch.fft.rfft((mass * self.pm).view(nr, nz, na), dim=2)[..., self.m]
        if self.nd == 3:
            s = torch.fft.fft(s, n=2 * nz, dim=1)
        s = s.permute(2, 1, 0).unsqueeze(-1)                                # [m, kz, is, 1]
        comp = {}
        for t, K in self.K.items():
            f = torch.matmul(K, s).squeeze(-1).permute(2, 1, 0)             # [ir, kz, m]
            if self.nd == 3:
                f = torch.fft.ifft(f, dim=1)[:, :nz]
            full = torch.zeros(nr, nz, na // 2 + 1, dtype=torch.complex128, device="cuda")
            full = full.index_copy(2, torch.tensor(self.m, device="cuda"), f)
            comp[t] = torch.fft.irfft(full, n=na, dim=2)
        fx = comp["r"] * self.cos - comp["t"] * self.sin
        fy = comp["r"] * self.sin + comp["t"] * self.cos
        return torch.stack([fx, fy] + [comp[t] for t in comp if t in "zp"], -1).view(nr * nz * na, -1)

    def force(self, x, cell, F):
        """Acceleration (and the grid's and halo's potential) at x."""
        on, idx, wt = cell
        a = sum(F[idx[:, k]] * wt[:, k:k + 1] for k in range(idx.shape[1]))
        acc, pot = a[:, :self.nd], a[:, self.nd] if a.shape[1] > self.nd else None
        if self.halo:
            g = on.to(torch.float64)
            d = x.square().sum(1) + self.rc ** 2
            k = self.v2 / d if self.halo == 1 else self.v2 * d ** -1.5
            acc = acc - (k * g)[:, None] * x
            if pot is not None:
                pot = pot + g * (0.5 * self.v2 * torch.log(d / self.rc ** 2) if self.halo == 1 else -self.v2 * d ** -0.5)
        return acc, pot

    def step(self, x, v):
        cell = self.cells(x)
        a, _ = self.force(x, cell, self.field(self.mass(cell)))
        v = v + a
        return x + v, v

    def zoned(self, rec, steps, nstep, zbr):
        """The reference's time-step zones: each zone steps at its own multiple
        of the base step and keeps the masses of its last two positions, which
        the solve interpolates in time."""
        nd, nz = self.nd, len(nstep)
        x, v = rec[:, :nd].clone(), rec[:, nd:].clone()
        fac = torch.tensor([float(s) for s in nstep] + [float(nstep[-1])], device="cuda", dtype=torch.float64)
        edges = torch.tensor([float(np.float32(b)) for b in zbr[1:]], device="cuda", dtype=torch.float64)
        def zone_of(x): return (x.square().sum(1).sqrt()[:, None] >= edges[None]).sum(1)
        on = self.cells(x)[0]
        zone = torch.where(on, zone_of(x), torch.full_like(on, nz, dtype=torch.long))
        v = v * torch.where(on, fac[zone], torch.ones_like(fac[zone]))[:, None]
        def masses(which): return self.mass_of(x, zone == which)
        new = [masses(k) for k in range(nz)]
        old, tnew, told = list(new), [0] * nz, [0] * nz
        for i in range(steps):
            m = new[0].clone()
            for k in range(1, nz):
                w = (tnew[k] - i) / nstep[k]
                m = m + ((1 - w) * new[k] + (w * old[k] if w else 0))
            F = self.field(m)
            top = max(k for k in range(nz) if i % nstep[k] == 0)
            move = (zone <= top) | ((zone == nz) & (top == nz - 1))
            a, _ = self.force(x, self.cells(x), F)
            t = fac[zone][:, None]
            a = torch.where((zone < nz)[:, None], a * t * t, torch.zeros_like(a))
            xo, vo = x, v
            vn = vo + a
            xn = xo + vn
            def redo(sel, f, xn, vn, a):
                s = sel[:, None]
                f = f[:, None]
                v2 = f * (vo + 0.5 * a * (1 - f))
                a2 = a * f * f
                v2 = v2 + a2
                return torch.where(s, xo + v2, xn), torch.where(s, v2, vn), torch.where(s, a2, a)
            on = self.cells(xn)[0]
            left = (zone < nz) & ~on
            zn = torch.where(left, nz, torch.where((zone == nz) & on, nz - 1, zone))
            xn, vn, a = redo(left & (zone < nz - 1), fac[nz - 1] / fac[zone], xn, vn, a)
            if top > 0:
                k = zone_of(xn).clamp(max=top)
                k = torch.where(k > zn, zone_of(xo), k)
                ch = (zone < nz) & (zn <= top) & (k != zn)
                xn, vn, a = redo(ch, fac[k] / fac[zn], xn, vn, a)
                zn = torch.where(ch, k, zn)
            x = torch.where(move[:, None], xn, x)
            v = torch.where(move[:, None], vn, v)
            zone = torch.where(move, zn, zone)
            for k in range(top + 1):
                old[k], told[k] = new[k], tnew[k]
                new[k], tnew[k] = masses(k), i + nstep[k]
        return torch.cat([x, torch.where((zone < nz)[:, None], v / fac[zone][:, None], v)], 1)

    def mass_of(self, x, sel):
        on, idx, wt = self.cells(x)
        return self.mass((on, idx, wt * sel.to(torch.float64)[:, None]))


class Disc:
    """Functions U_nm of the Abel-Jacobi basis (and their derivatives) in FP64."""

    def __init__(self, c):
        d = json.load(open(BASIS))
        self.c, self.k = c, d["k"]
        self.roots = {tuple(int(q) for q in k.split(",")): v for k, v in d["roots"].items()}
        self.xc = {tuple(int(q) for q in k.split(",")): v for k, v in d["xcoeff"].items()}
        self.front = math.pi / float(np.float32(math.sqrt(2.0)))

    def radial(self, m, p, der):
        """Yield (n, U, dU/dp) for every n, p in [0, 1]."""
        p2, s = p * p, 1 - p * p
        pm = p ** m if m else torch.ones_like(p)
        dpm = m * p ** (m - 1) if m else torch.zeros_like(p)
        for n in range(self.c["maxn"] + 1):
            xc = self.xc[(m, n)]
            f, g = torch.full_like(p, xc[-1]), torch.zeros_like(p)
            for q in xc[-2::-1]:
                if der:
                    g = g * s + f
                f = f * s + q
            g = g * (-2 * p)
            for rt in self.roots[(m, n)][:n]:
                b = p2 - rt * rt
                if der:
                    g = g * b + f * (2 * p)
                f = f * b
            yield n, self.front * pm * f, self.front * (pm * g + dpm * f) if der else None

    def coeff(self, x, pmass, maxr):
        rr = x.square().sum(1).sqrt()
        x = x[rr <= maxr]
        rr = rr[rr <= maxr]
        p, ph = rr / maxr, torch.atan2(x[:, 1], x[:, 0])
        mm, nn = self.c["maxm"], self.c["maxn"]
        out = torch.zeros(nn + 1, 2 * mm + 1, dtype=torch.float64, device="cuda")
        for m in range(mm + 1):
            cs, sn = (m * ph).cos(), (m * ph).sin()
            for n, U, _ in self.radial(m, p, False):
                out[n, mm + m] = (U * cs).sum()
                if m:
                    out[n, mm - m] = (U * sn).sum()
        return out * (pmass / maxr ** 2)

    def acc(self, x, coeff, maxr):
        """-grad of the potential of the coefficients, per particle."""
        rr = x.square().sum(1).sqrt()
        on = (rr <= maxr).to(torch.float64)
        r = rr.clamp(min=1e-5)
        p, ph = (rr / maxr).clamp(max=1.0), torch.atan2(x[:, 1], x[:, 0])
        mm = self.c["maxm"]
        ar, at = torch.zeros_like(r), torch.zeros_like(r)
        for m in range(mm + 1):
            cs, sn = (m * ph).cos(), (m * ph).sin()
            fc, fs, dc, ds = (torch.zeros_like(r) for _ in range(4))
            for n, U, D in self.radial(m, p, True):
                a, b = coeff[n, mm + m], coeff[n, mm - m] if m else 0.0
                fc, dc = fc + a * U, dc + a * D
                if m:
                    fs, ds = fs + b * U, ds + b * D
            ar = ar + dc * cs + ds * sn
            at = at + m * (fs * cs - fc * sn)
        at = at * (maxr / r)
        c1, s1 = x[:, 0] / r, x[:, 1] / r
        return torch.stack([ar * c1 - at * s1, ar * s1 + at * c1], 1) * on[:, None]


def exact(case, seed):
    c = case
    if c["kind"].startswith("sfp"):
        rec, d = _exp_disc(c["n"], seed).double(), Disc(c)
        x, v = rec[:, :2], rec[:, 2:]
        if c["kind"] == "sfp_sum":
            return {"coeff": d.coeff(x, 1.0 / c["n"], 6.0)}
        dt = float(np.float32(0.01))
        for _ in range(c["steps"]):
            v = v + d.acc(x, d.coeff(x, 1.0 / c["n"], 6.0), 6.0) * dt
            x = x + v * dt
        return {"coeff": d.coeff(x, 1.0 / c["n"], 6.0), "particles": torch.cat([x, v], 1)}
    if c["kind"] == "ensemble":
        out, K = [], None
        for k, n in enumerate(_counts(c)):
            rec, pm = _disc(c, int(n), seed * 1000 + k)
            if K is None:
                K = Mesh(c, pm)
            K.pm = float(np.float32(pm))
            x, v = rec[:, :2].double(), rec[:, 2:].double()
            for _ in range(c["steps"]):
                x, v = K.step(x, v)
            out.append(torch.cat([x, v], 1))
        return {"particles": out}
    rec, pm = _disc(c, c["n"], seed)
    rec, nd = rec.double(), c["ndim"]
    M = Mesh(c, pm, pot=c["kind"] == "forces")
    x, v = rec[:, :nd], rec[:, nd:]
    if c["kind"] == "forces":
        cell = M.cells(x)
        acc, pot = M.force(x, cell, M.field(M.mass(cell)))
        return {"acc": acc, "pot": pot}
    if c["kind"] == "zones":
        return {"particles": M.zoned(rec, c["steps"], *_zones(c))}
    if c["kind"] == "run":
        for _ in range(c["steps"]):
            x, v = M.step(x, v)
        return {"particles": torch.cat([x, v], 1)}
    # the gradient by automatic differentiation of the same steps
    x0, v0 = x.clone().requires_grad_(), v.clone().requires_grad_()
    M.rc.requires_grad_()
    M.v2.requires_grad_()
    x, v = x0, v0
    for _ in range(c["steps"]):
        x, v = torch.utils.checkpoint.checkpoint(M.step, x, v, use_reentrant=False)
    r2 = x.square().sum(1)
    re = ((x[:, 0] ** 2 - x[:, 1] ** 2) / r2).mean()
    im = (2 * x[:, 0] * x[:, 1] / r2).mean()
    J = (re * re + im * im).sqrt()
    J.backward()
    zero = torch.zeros((), dtype=torch.float64, device="cuda")
    dth = torch.stack([zero if q.grad is None else q.grad for q in (M.rc, M.v2)])
    return {"J": J.detach(), "grad": torch.cat([x0.grad, v0.grad], 1), "dtheta": dth}
