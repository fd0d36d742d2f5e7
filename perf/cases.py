"""Workloads of the semi-Lagrangian advection path, as a host model runs them.

Each case is one pass of a time step, or of one of the passes that follow the
interpolation of the tracers, through the public entry points of
``gem_b200.adz`` and ``gem_b200.guess``:

  step    one whole advection step: departure points from the previous step's,
          then u, v, w and every tracer interpolated at their position sets
  cold    the first step of a run: network start, iteration to a tolerance,
          then the interpolations
  qv      tracers interpolated with BICUBH_QV and their bounds
  fixer   tracers interpolated with bounds, LAM boundary fluxes, then the
          Bermejo-Conde mass fixer
  ilmc    tracers interpolated with bounds, then the ILMC filter
  interp  the reference's monotone interpolator on explicit positions
  batch   one step of many small independent domains

Grids, flows, noise and tracers are those of ``gem_b200.synth``.
"""
import math

import numpy as np
import torch

from gem_b200 import adz as A
from gem_b200 import guess as G
from gem_b200 import synth

SLT_EPS = 2.0e-5
WIND_KEYS = ("uu_ext", "vv_ext", "ww_ext", "ut0", "vt0", "zdt0")


def listed():
    return [
        # the headline tile of the benchmark: 1024 x 1024 x 80, u, v, w and 4 cosine bells
        dict(name="step_mixed_large", kind="step", prec="mixed", ni=1024, nj=1024, nk=80, ntr=4, tracer="bells",
             mono=False, dt=60.0, dx=2500.0, u0=40.0, cap=1000.0),
        # a chemistry run on an odd-sized tile of a decomposition: 8 monotone log-normal tracers
        dict(name="step_mixed_tracers", kind="step", prec="mixed", ni=509, nj=387, nk=80, ntr=8, tracer="lognormal",
             mono=True, dt=60.0, dx=2500.0, u0=40.0, cap=1000.0),
        # the smallest configuration of the tests and the benchmark: launches and tails count
        dict(name="step_mixed_small", kind="step", prec="mixed", ni=128, nj=128, nk=40, ntr=2, tracer="bell+uniform",
             mono=False, dt=300.0, dx=10000.0, u0=40.0, cap=0.0),
        # the FP64 drop-in
        dict(name="step_fp64", kind="step", prec="fp64", ni=640, nj=512, nk=80, ntr=4, tracer="bells", mono=False,
             dt=60.0, dx=2500.0, u0=40.0, cap=1000.0),
        # the reference's own arithmetic, bit for bit, on a ragged tile
        dict(name="step_ref32", kind="step", prec="ref32", ni=451, nj=393, nk=61, ntr=3, tracer="lognormal",
             mono=True, dt=120.0, dx=2500.0, u0=30.0, cap=1000.0),
        # first step of a run: no previous departure points
        dict(name="cold_mixed", kind="cold", prec="mixed", ni=768, nj=640, nk=80, ntr=4, tracer="bells", mono=False,
             dt=60.0, dx=2500.0, u0=40.0, cap=1000.0),
        # tracers of a run that interpolates them with the quintic scheme
        dict(name="qv_mixed", kind="qv", prec="mixed", ni=640, nj=600, nk=80, ntr=8, tracer="lognormal", mono=True,
             dt=60.0, dx=2500.0, u0=40.0, cap=1000.0),
        # tracer mass conservation of a limited-area run
        dict(name="fixer_mixed", kind="fixer", prec="mixed", ni=640, nj=600, nk=80, ntr=4, tracer="lognormal",
             mono=True, dt=60.0, dx=2500.0, u0=40.0, cap=1000.0),
        # the same, shape-preserving filter instead, in the reference's arithmetic
        dict(name="ilmc_ref32", kind="ilmc", prec="ref32", ni=301, nj=262, nk=80, ntr=3, tracer="lognormal",
             mono=True, dt=60.0, dx=2500.0, u0=40.0, cap=1000.0),
        # a caller that computes its own positions and links the interpolator only
        dict(name="interp_ref32", kind="interp", prec="ref32", ni=600, nj=400, nk=58, ntr=5, tracer="lognormal",
             mono=True, dt=60.0, dx=2500.0, u0=40.0, cap=1000.0),
        # an ensemble of small limited-area domains advanced together
        dict(name="batch_mixed", kind="batch", prec="mixed", ni=96, nj=112, nk=50, ntr=4, tracer="lognormal",
             mono=True, dt=120.0, dx=2500.0, u0=40.0, cap=1000.0, domains=24),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["step"] * 5 + ["cold", "qv", "fixer", "ilmc", "interp", "batch"])
    prec = rng.choice(["mixed", "mixed", "fp64", "ref32"])
    hi = 900
    c = dict(kind=kind, ntr=rng.randint(1, 8))
    if kind == "cold":
        prec, hi = "mixed", 700
    elif kind == "batch":
        prec, hi = rng.choice(["mixed", "fp64"]), 150
        c["domains"] = rng.randint(4, 32)
    elif kind == "ilmc":
        hi = 260
        c["ntr"] = rng.randint(1, 3)
    elif kind in ("fixer", "interp"):
        hi = 600
        c["ntr"] = rng.randint(1, 6)
    elif prec == "fp64":
        hi = 640
    lo = 48 if kind == "batch" else 64
    u0 = round(rng.uniform(20.0, 60.0), 2)
    dt = round(rng.uniform(60.0, 300.0), 1) if kind != "cold" else round(rng.uniform(60.0, 120.0), 1)
    # Courant numbers up to about 2, as in a run with dt chosen for its grid
    c.update(prec=prec, ni=log(lo, hi), nj=log(lo, hi), nk=rng.randint(24, 80), u0=u0, dt=dt,
             dx=round(max(2500.0, u0 * dt / rng.uniform(0.8, 2.0)), 1), mono=rng.random() < 0.6 or kind in (
                 "qv", "fixer", "ilmc", "interp"), tracer=rng.choice(["lognormal", "bells", "bell+uniform"]),
             cap=rng.choice([0.0, 1000.0]))
    return c


# ---------------------------------------------------------------------------
def _levels(case):
    if case["cap"] > 0:
        return synth.stretched_levels(case["nk"], 20.0, max(case["cap"], 1.05 * 25e3 / case["nk"]), 25e3)
    return synth.uniform_levels(case["nk"], 20e3)


def _config(case, seed, part=0):
    """One synthetic domain; domains of a batch differ in size and phase."""
    rng = np.random.default_rng([int(seed), 77, part])
    sizes = np.random.default_rng([case["ni"], case["nj"], part])  # sizes belong to the case, not to the seed
    ni, nj, nk = case["ni"], case["nj"], case["nk"]
    ntr = case["ntr"]
    if case["kind"] == "batch":
        ni = max(40, int(ni * sizes.uniform(0.5, 1.5)))
        nj = max(40, int(nj * sizes.uniform(0.5, 1.5)))
        ntr = int(sizes.integers(1, ntr + 1))
    lev = _levels(case)
    # W0 and the noise keep the vertical displacement of a step at some tens
    # of metres (some layers, near the ground)
    w0 = 30.0 / case["dt"]
    return synth.Config(case["kind"], ni, nj, nk, case["dx"], case["dt"], lev, niter=2, u0=case["u0"], w0=w0,
                        noise_w=0.02 if case["kind"] == "cold" else min(0.5, 30.0 / case["dt"]),
                        seed=int(seed) * 131 + part, ntracers=ntr, tracer_kind=case["tracer"],
                        bell_radius=0.2 * ni * case["dx"], mono=case["mono"],
                        phase=(float(rng.uniform(0, 1)), float(rng.uniform(0, 1))))


def _inputs(cfg, prec):
    return synth.make_inputs(cfg, device="cuda", dtype=A._field_dtype(A.PREC_NAMES[prec]))


def _start(cfg, inp, prec):
    """Departure points of the previous step, as its trajectory leaves them:
    winds at the arrival point over one time step.  Returns wpxyz and, for
    REF32, pxyzm."""
    H, ni, nj, nk = cfg.halo, cfg.ni, cfg.nj, cfg.nk
    c = (slice(None), slice(H, H + nj), slice(H, H + ni))
    f64 = torch.float64
    i = torch.arange(1, ni + 1, device="cuda", dtype=f64)
    j = torch.arange(1, nj + 1, device="cuda", dtype=f64)
    wp = torch.zeros((3, nk, nj + 4, ni + 4), dtype=f64, device="cuda")
    x, y, z = (wp[q, :, 2:nj + 2, 2:ni + 2] for q in range(3))
    x.copy_(i - 0.5 * cfg.dt / cfg.dx * (inp["uu_ext"][c].to(f64) + inp["ut0"][c]))
    y.copy_(j.view(-1, 1) - 0.5 * cfg.dt / cfg.dx * (inp["vv_ext"][c].to(f64) + inp["vt0"][c]))
    zm = torch.tensor(cfg.levels.zm, device="cuda", dtype=f64)
    pos = zm[1:nk + 1].view(-1, 1, 1) - 0.5 * cfg.dt * (inp["ww_ext"][c].to(f64) + inp["zdt0"][c])
    z.copy_(_height_index(pos, zm, nk))
    px = None
    if prec == "ref32":
        b = _bounds(cfg)
        px = torch.stack([x.clamp(b[0], b[1]), y.clamp(b[2], b[3]), z], dim=-1).to(torch.float32).contiguous()
    return wp, px


def prepare(case, seed):
    kind, prec = case["kind"], A.PREC_NAMES[case["prec"]]
    ft = A._field_dtype(prec)
    if kind == "batch":
        doms = []
        for p in range(case["domains"]):
            cfg = _config(case, seed, p)
            inp = _inputs(cfg, case["prec"])
            ad = A.Adz.from_config(cfg)
            px, wp = ad.new_state(prec)
            ad.adz_inittraj(prec, px, wp)
            ad.adz_traject(prec, cfg.dt, inp, px, wp)
            wp.copy_(_start(cfg, inp, case["prec"])[0])
            srcs = [inp["src_u"], inp["src_v"], inp["src_w"]] + inp["tracers"]
            dsts = [torch.zeros(ad.ext_shape, dtype=ft, device="cuda") for _ in srcs]
            doms.append(dict(adz=ad, dt=cfg.dt, winds=inp, wpxyz=wp, nfields=[0, 1, 1, len(srcs) - 2], srcs=srcs,
                             dsts=dsts, mono=[0, 0, 0] + [int(case["mono"])] * (len(srcs) - 3)))
        torch.cuda.synchronize()
        b = A.Batch(prec, doms)
        start = [d["wpxyz"].clone() for d in doms]
        b.tune()
        for d, w in zip(doms, start):  # the tuner's timed steps moved the departure points
            d["wpxyz"].copy_(w)
        return dict(kind=kind, batch=b, doms=doms)
    cfg = _config(case, seed)
    inp = _inputs(cfg, case["prec"])
    if kind == "interp":
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        H, n = cfg.halo, (cfg.ni - 16) * (cfg.nj - 16) * 6
        wp, px = _start(cfg, inp, "ref32")
        k = cfg.nk // 2
        pos = px[k - 3:k + 3, 8:-8, 8:-8].reshape(n, 3).contiguous()
        zt = A.Ztab(cfg.levels.zt[1:cfg.nk + 1], cfg.ni + 2 * H, cfg.nj + 2 * H, 0, 0)
        if case["prec"] != "ref32":
            pos = pos.double() + 1e-9 * torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)
        at = H * (cfg.ni + 2 * H) + H  # element (1, 1, 1) of an extended array
        return dict(kind=kind, zt=zt, prec=prec, pos=pos, ext=inp["tracers"],
                    srcs=[t.view(-1)[at:] for t in inp["tracers"]])
    ad = A.Adz.from_config(cfg)
    new = lambda: torch.zeros(ad.ext_shape, dtype=ft, device="cuda")  # noqa: E731
    tracers = inp["tracers"]
    st = dict(kind=kind, prec=prec, cfg=cfg, ad=ad, inp=inp, tracers=tracers, tr_outs=[new() for _ in tracers],
              mono=case["mono"])
    if kind == "cold":
        st.update(net=G.GuessNet(), wp=ad.new_state(prec)[1], outs={q: new() for q in "uvw"})
        return st
    wp, px = _start(cfg, inp, case["prec"])
    st.update(wp=wp, px=px)
    if kind == "step":
        st["outs"] = {q: new() for q in "uvw"}
        return st
    # the passes after the trajectory start from its departure points
    ad.adz_traject(prec, cfg.dt, inp, px, wp)
    st["post"] = tuple([new() for _ in tracers] for _ in range(3))
    if kind in ("fixer", "ilmc"):
        g = torch.Generator(device="cuda").manual_seed(int(seed) + 5)
        rnd = lambda *s: torch.rand(s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
        ap = 1.0 + 0.2 * rnd(*ad.ext_shape)
        st["air_p"] = ap.to(ft)
        st["air_m"] = (ap * (1.0 + 0.01 * rnd(*ad.ext_shape))).to(ft)
        st["mask"] = cfg.dx ** 2 * (0.5 + rnd(cfg.nj, cfg.ni))
    if kind == "fixer":
        st.update(fo=[new() for _ in tracers], fi=[new() for _ in tracers])
    return st


def run(s):
    kind = s["kind"]
    if kind == "batch":
        s["batch"].step()
        return [dict(wpxyz=d["wpxyz"], fields=d["dsts"]) for d in s["doms"][:8]]
    if kind == "interp":
        d, lin, mn, mx = A.tricublin_mono_m_n(s["zt"], s["prec"], s["srcs"], s["pos"])
        return dict(d=d, lin=lin, mn=mn, mx=mx)
    ad, prec, inp, cfg = s["ad"], s["prec"], s["inp"], s["cfg"]
    if kind == "step":
        A.step_fused(ad, prec, cfg.dt, inp, inp, s["tracers"], s["px"], s["wp"], s["outs"], s["tr_outs"], s["mono"])
        out = dict(s["outs"], tracers=s["tr_outs"], wpxyz=s["wp"])
        if s["px"] is not None:
            out["pxyzm"] = s["px"]
        return out
    if kind == "cold":
        G.traject_guess(ad, s["net"], cfg.dt, inp, s["wp"], stride=16)
        srcs = [inp["src_u"], inp["src_v"], inp["src_w"]] + s["tracers"]
        dsts = [s["outs"]["u"], s["outs"]["v"], s["outs"]["w"]] + s["tr_outs"]
        ad.adz_tricub_sets(prec, [0, 1, 1, 1 + len(s["tracers"])], srcs, dsts,
                           [0, 0, 0] + [int(s["mono"])] * len(s["tracers"]))
        return dict(s["outs"], tracers=s["tr_outs"], wpxyz=s["wp"])
    n = len(s["tracers"])
    lin, mn, mx = s["post"]
    if kind == "qv":
        ad.adz_tricub_hlt(prec, A.SET_T, s["tracers"], s["tr_outs"], mono=[A.QV | 1] * n, post=s["post"])
        return dict(tracers=s["tr_outs"], lin=lin, mn=mn, mx=mx)
    ad.adz_tricub_hlt(prec, A.SET_T, s["tracers"], s["tr_outs"], mono=[2] * n, post=s["post"])
    if kind == "ilmc":
        A.ilmc(ad, prec, s["tr_outs"], mn, mx, s["air_m"])
        return dict(tracers=s["tr_outs"])
    ad.bc_lam_flux(prec, s["tracers"], s["fo"], s["fi"])
    deficit = torch.zeros(n, dtype=torch.float64, device="cuda")
    tr = [dict(p=s["tracers"][q], m=s["tr_outs"][q], lin=lin[q], min=mn[q], max=mx[q], fo=s["fo"][q], fi=s["fi"][q])
          for q in range(n)]
    # the masses come back in diag; the deficit left over is their rounding
    diag = torch.zeros((n, 8), dtype=torch.float64, device="cuda")
    A.bermejo_conde(ad, prec, tr, s["air_p"], s["air_m"], s["mask"], deficit, diag=diag)
    return dict(tracers=s["tr_outs"], fo=s["fo"], fi=s["fi"], diag=diag)


# ---------------------------------------------------------------------------
def work(case):
    """Every input read once and every output written once; the flops of the
    stencil sums (a cubic value: 64 + 16 + 4 multiply-adds)."""
    fb = 8 if case["prec"] == "fp64" else 4
    pts = float(case["ni"] * case["nj"] * case["nk"])
    n, kind = case["ntr"], case["kind"]
    if kind == "batch":
        pts = ntot = 0.0
        for p in range(case["domains"]):
            c = _config(case, 0, p)
            pts += c.npoints
            ntot += c.npoints * (3 + c.ntracers)
        return dict(bytes=pts * (6 * fb + 48) + 2 * fb * ntot, flops=pts * 2 * 650 + 168 * ntot)
    if kind == "step":
        start = 24 + (24 if case["prec"] == "ref32" else 24)
        return dict(bytes=pts * (6 * fb + start + 2 * fb * (3 + n)), flops=pts * (2 * 650 + 168 * (3 + n)))
    if kind == "cold":
        return dict(bytes=pts * (6 * fb + 24 + 2 * fb * (3 + n)), flops=pts * (2.5 * 650 + 168 * (3 + n)))
    if kind == "interp":
        m = float((case["ni"] - 16) * (case["nj"] - 16) * 6)
        src = float(case["ni"] * case["nj"] * 12) * fb * n
        return dict(bytes=m * ((12 if case["prec"] == "ref32" else 24) + 4 * fb * n) + src, flops=m * 220 * n)
    pos = 28 + 2 * fb  # departure points and vertical winds of the t set
    if kind == "qv":
        return dict(bytes=pts * (pos + 5 * fb * n), flops=pts * 300 * n)
    if kind == "ilmc":  # interpolation with bounds, then the fields and bounds once more
        return dict(bytes=pts * (pos + 5 * fb * n + (4 * n + 1) * fb), flops=pts * 240 * n)
    # fixer: interpolation with bounds; two fluxes; masses, correction, rescale
    return dict(bytes=pts * (pos + 5 * fb * n + 3 * fb * n + (9 * n + 2) * fb), flops=pts * (220 + 2 * 168) * n)


def tolerance(case):
    """REF32 and FP64 reproduce the reference's operation order; the fixer's
    sums may add up in another one.  MIXED sums in FP32: its fields are 1e-7
    from the 64-bit ones, and the rounding of a trajectory moves a departure
    point by some 1e-6 grid lengths, which single values of white-noise
    tracers show as 1e-4 of their magnitude.  The ILMC filter decides by sign
    which points it touches."""
    kind, prec = case["kind"], case["prec"]
    if prec == "mixed":
        return {"rel": 1e-5, "max": 0.05} if kind == "ilmc" else {"rel": 5e-7, "max": 1e-3}
    if kind == "fixer":
        return {"rel": 5e-7 if prec == "ref32" else 1e-12, "max": 1e-5 if prec == "ref32" else 1e-10}
    return "exact"


# ---------------------------------------------------------------------------
# the same values in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _bounds(cfg):
    """Clip bounds of departure points in a domain that touches all edges."""
    return (5 + SLT_EPS, cfg.ni - 4 - SLT_EPS, 5 + SLT_EPS, cfg.nj - 4 - SLT_EPS)


def _height_index(pos, z, nk):
    """Fractional level index of heights (levels z[0..nk+1], descending)."""
    pos = pos.clamp(float(z[nk + 1]), float(z[0]))
    nb = (torch.searchsorted(-z, -pos.contiguous(), right=True) - 1).clamp(1, nk - 1)
    return (pos - z[nb]) / (z[nb + 1] - z[nb]) + nb


def _lag(x, nodes, q):
    w = None
    for r, n in enumerate(nodes):
        if r != q:
            f = (x - n) / (nodes[q] - n)
            w = f if w is None else w * f
    return w


def _lag3(x, a, b, c, d):
    """Weight of node a of the cubic through a, b, c, d at x."""
    return (x - b) * (x - c) * (x - d) / ((a - b) * (a - c) * (a - d))


class _Exact:
    def __init__(self, cfg):
        self.cfg, self.H = cfg, cfg.halo
        self.ni, self.nj, self.nk = cfg.ni, cfg.nj, cfg.nk
        self.nit, self.njt = cfg.ni + 2 * self.H, cfg.nj + 2 * self.H
        t = lambda a: torch.tensor(a, device="cuda", dtype=torch.float64)  # noqa: E731
        self.zm, self.zt, self.zx = t(cfg.levels.zm), t(cfg.levels.zt), t(cfg.levels.zx)
        self.b = _bounds(cfg)
        self.dth = 0.5 * cfg.dt

    def clip(self, x, y):
        return x.clamp(self.b[0], self.b[1]), y.clamp(self.b[2], self.b[3])

    def cells(self, p, lo=None, hi=None):
        c = p.float().to(torch.int64)  # truncation of the 32-bit rounding
        if lo is not None:
            c = c.clamp(lo, hi)
        return c, p - c

    def stencil(self, px, py, pz, z):
        ix, tx = self.cells(px)
        iy, ty = self.cells(py)
        iz, tz = self.cells(pz, 1, self.nk - 1)
        cub = (iz >= 2) & (iz <= self.nk - 2)
        h = z[iz] + tz * (z[iz + 1] - z[iz])
        izc = torch.where(cub, iz, torch.full_like(iz, 2))
        hc = torch.where(cub, h, z[izc])
        nodes = [z[izc - 1 + q] for q in range(4)]
        lin = [torch.zeros_like(tz), 1 - tz, tz, torch.zeros_like(tz)]
        wz = [torch.where(cub, _lag(hc, nodes, q), lin[q]) for q in range(4)]
        wx = [_lag(tx, (-1.0, 0.0, 1.0, 2.0), q) for q in range(4)]
        wy = [_lag(ty, (-1.0, 0.0, 1.0, 2.0), q) for q in range(4)]
        base = (ix - 2 + self.H) + (iy - 2 + self.H) * self.nit
        planes = [(iz - 2 + q).clamp(0, self.nk - 1) * (self.nit * self.njt) for q in range(4)]
        return dict(wx=wx, wy=wy, wz=wz, base=base, planes=planes, tx=tx, ty=ty, tz=tz)

    def cubic(self, f, s, mono=False):
        f = f.reshape(-1)
        out = torch.zeros_like(s["tx"])
        lin = torch.zeros_like(out)
        mn, mx = torch.full_like(out, math.inf), torch.full_like(out, -math.inf)
        for p in range(4):
            for r in range(4):
                for x in range(4):
                    v = f[s["base"] + s["planes"][p] + (r * self.nit + x)].to(torch.float64)
                    out += v * (s["wz"][p] * s["wy"][r] * s["wx"][x])
                    if mono and p in (1, 2) and x in (1, 2):
                        mn, mx = torch.minimum(mn, v), torch.maximum(mx, v)
                        if r in (1, 2):
                            w = (s["tx"] if x == 2 else 1 - s["tx"]) * (s["ty"] if r == 2 else 1 - s["ty"])
                            lin += v * w * (s["tz"] if p == 2 else 1 - s["tz"])
        return (out, lin, mn, mx) if mono else out

    def quintic(self, f, px, py, pz):
        nk, z, f = self.nk, self.zt, f.reshape(-1)
        ix, tx = self.cells(px)
        iy, ty = self.cells(py)
        iz = pz.float().to(torch.int64)
        q5, q3 = (iz >= 3) & (iz <= nk - 3), (iz == 2) | (iz == nk - 2)
        iz = torch.where(q5 | q3, iz, iz.clamp(1, nk - 1))
        tz = pz - iz
        h = z[iz] + tz * (z[iz + 1] - z[iz])
        tl = (h - z[iz]) / (z[iz + 1] - z[iz])
        i5, i3 = torch.where(q5, iz, torch.full_like(iz, 3)), torch.where(q3, iz, torch.full_like(iz, 2))
        n5, n3 = [z[i5 - 2 + q] for q in range(6)], [z[i3 - 1 + q] for q in range(4)]
        h5, h3 = torch.where(q5, h, z[i5]), torch.where(q3, h, z[i3])
        zero = torch.zeros_like(tl)
        w3 = [zero] + [_lag(h3, n3, q) for q in range(4)] + [zero]
        wl = [zero, zero, 1 - tl, tl, zero, zero]
        wz = [torch.where(q5, _lag(h5, n5, q), torch.where(q3, w3[q], wl[q])) for q in range(6)]
        wx = [_lag(tx, (-1.0, 0.0, 1.0, 2.0), q) for q in range(4)]
        wy = [_lag(ty, (-1.0, 0.0, 1.0, 2.0), q) for q in range(4)]
        base = (ix - 2 + self.H) + (iy - 2 + self.H) * self.nit
        out, lin = torch.zeros_like(px), torch.zeros_like(px)
        mn, mx = torch.full_like(px, math.inf), torch.full_like(px, -math.inf)
        for p in range(6):
            plane = (iz - 3 + p).clamp(0, nk - 1) * (self.nit * self.njt)
            for r in range(4):
                for x in range(4):
                    v = f[base + plane + (r * self.nit + x)].to(torch.float64)
                    out += v * (wz[p] * wy[r] * wx[x])
                    if p in (2, 3) and r in (1, 2) and x in (1, 2):
                        mn, mx = torch.minimum(mn, v), torch.maximum(mx, v)
                        lin += v * ((tx if x == 2 else 1 - tx) * (ty if r == 2 else 1 - ty) * (tl if p == 3 else 1 - tl))
        return out, lin, mn, mx

    def w_momentum(self, w):
        """Vertical wind on momentum levels from thermo levels."""
        nk, zx, zm = self.nk, self.zx, self.zm
        w = w.to(torch.float64)
        out = torch.empty_like(w)
        out[0] = (zx[0] - zm[1]) / (zx[0] - zx[1]) * w[0]
        out[nk - 1] = (zm[nk] - zx[nk]) / (zx[nk - 1] - zx[nk]) * w[nk - 2]
        for k in range(2, nk):
            a, b, c, d = (zx[k + q] for q in (-2, -1, 0, 1))
            v = _lag3(zm[k], b, a, c, d) * w[k - 2] + _lag3(zm[k], c, a, b, d) * w[k - 1] + _lag3(
                zm[k], d, a, b, c) * w[k]
            if k >= 3:
                v = v + _lag3(zm[k], a, b, c, d) * w[k - 3]
            out[k - 1] = v
        return out

    def trajectory(self, inp, start, niter):
        """Departure points of every point and the departure vertical wind."""
        H, ni, nj, nk, dx, h = self.H, self.ni, self.nj, self.nk, self.cfg.dx, self.dth
        uu, vv, ww = inp["uu_ext"], inp["vv_ext"], self.w_momentum(inp["ww_ext"])
        c = lambda f, di=0, dj=0: f[:, H + dj:H + dj + nj, H + di:H + di + ni].to(torch.float64)  # noqa: E731
        ut, vt = inp["ut0"], inp["vt0"]
        ua = (c(ut, -2) + c(ut, 1)) * (-1 / 16) + (c(ut) + c(ut, -1)) * (9 / 16)
        va = (c(vt, 0, -2) + c(vt, 0, 1)) * (-1 / 16) + (c(vt) + c(vt, 0, -1)) * (9 / 16)
        wa = c(self.w_momentum(inp["zdt0"]))
        i = torch.arange(1, ni + 1, device="cuda", dtype=torch.float64)
        j = torch.arange(1, nj + 1, device="cuda", dtype=torch.float64).view(-1, 1)
        dep, wdep = torch.empty((3, nk, nj, ni), device="cuda", dtype=torch.float64), torch.empty_like(wa)
        for k in range(0, nk, 4):
            kk = slice(k, k + 4)
            x, y = self.clip(start[0, kk], start[1, kk])
            z = start[2, kk].clone()
            for _ in range(niter):
                s = self.stencil(x, y, z, self.zm)
                ud, vd, wd = (self.cubic(f, s) for f in (uu, vv, ww))
                xm, ym = i - h * (ud + ua[kk]) / dx, j - h * (vd + va[kk]) / dx
                z = _height_index(self.zm[1:nk + 1].view(-1, 1, 1)[kk] - h * (wd + wa[kk]), self.zm, nk)
                x, y = self.clip(xm, ym)
            dep[0, kk], dep[1, kk], dep[2, kk], wdep[kk] = xm, ym, z, wd
        return dep, wdep

    def t_positions(self, dep, wdep, zd):
        """Departure points of the thermo levels, one level at a time (1..nk)."""
        H, nk, zm, zt = self.H, self.nk, self.zm, self.zt
        lev, dth = self.cfg.levels, self.dth
        zd = zd[:, H:H + self.nj, H:H + self.ni].to(torch.float64)
        wp = (lev.zt[nk] - lev.zm[nk - 1]) * lev.idz_t_nkm1

        def at(k):
            if 2 <= k <= nk - 2:
                n = [zm[k + q] for q in (-1, 0, 1, 2)]
                w = [_lag(zt[k], n, q) for q in range(4)]
                mix = lambda f: sum(w[q] * f[k - 2 + q] for q in range(4))  # noqa: E731
                z = zt[k] - dth * (mix(wdep) + zd[k - 1])
                return mix(dep[0]), mix(dep[1]), z
            if k == nk:
                mix = lambda f: wp * f[nk - 1] + (1 - wp) * f[nk - 2]  # noqa: E731
                z = zt[k] - lev.wmstar_nk * dth * (0.5 * (wdep[nk - 2] + wdep[nk - 1]) + zd[nk - 2])
                return mix(dep[0]), mix(dep[1]), z
            mix = lambda f: 0.5 * (f[k - 1] + f[k])  # noqa: E731
            return mix(dep[0]), mix(dep[1]), zt[k] - dth * (mix(wdep) + zd[k - 1])

        for k in range(1, nk + 1):
            x, y, z = at(k)
            x, y = self.clip(x, y)
            yield k, x, y, _height_index(z, zt, nk)

    def box(self, which):
        """First and last i, j of an arrival range (1-based), pilot zone 8."""
        p = self.cfg.pil
        b = dict(t=(p - 1, self.ni - p + 1, p - 1, self.nj - p + 1), u=(1 + p, self.ni - 1 - p, p - 1, self.nj - p + 1),
                 v=(p - 1, self.ni - p + 1, 1 + p, self.nj - 1 - p), core=(1 + p, self.ni - p, 1 + p, self.nj - p),
                 b=(5, self.ni - 4, 5, self.nj - 4))[which]
        return slice(b[2] - 1, b[3]), slice(b[0] - 1, b[1])

    def new(self):
        return torch.zeros((self.nk, self.njt, self.nit), device="cuda", dtype=torch.float64)

    def put(self, out, k, box, v):
        H = self.H
        out[k - 1, H:H + self.nj, H:H + self.ni][box] = v

    def t_set(self, tracers, dep, wdep, zd, how, clip, post=False, box="t"):
        """how: cubic, mono or qv; returns lists of extended arrays."""
        b = self.box(box)
        res = [[self.new() for _ in tracers] for _ in range(4 if post else 1)]
        for k, x, y, z in self.t_positions(dep, wdep, zd):
            x, y, z = x[b], y[b], z[b]
            s = None if how == "qv" else self.stencil(x, y, z, self.zt)
            for q, f in enumerate(tracers):
                if how == "cubic":
                    v, rest = self.cubic(f, s), ()
                else:
                    v, lin, mn, mx = self.quintic(f, x, y, z) if how == "qv" else self.cubic(f, s, True)
                    if clip:
                        v = torch.maximum(mn, torch.minimum(mx, v))
                    rest = (torch.maximum(mn, torch.minimum(mx, lin)), mn, mx)
                for o, a in zip(res, (v,) + tuple(rest)):
                    self.put(o[q], k, b, a)
        return res if post else res[0]

    def momentum(self, f, dep, which):
        """u or v at its staggered departure points."""
        b, out, nk = self.box(which), self.new(), self.nk
        ax = 1 if which == "u" else 0  # axis of a (nj, ni) plane
        for k in range(1, nk + 1):
            def mean(a):
                r = lambda n: torch.roll(a, -n, ax)  # noqa: E731
                return -0.0625 * (r(-1) + r(2)) + 0.5625 * (a + r(1))
            x, y, z = (mean(dep[q, k - 1]) for q in range(3))
            x, y = (x - 0.5, y) if which == "u" else (x, y - 0.5)
            x, y = self.clip(x, y)
            s = self.stencil(x[b], y[b], z.clamp(0.0, nk + 1.0)[b], self.zm)
            self.put(out, k, b, self.cubic(f, s))
        return out

    def fields(self, inp, dep, wdep, mono):
        out = dict(u=self.momentum(inp["src_u"], dep, "u"), v=self.momentum(inp["src_v"], dep, "v"))
        out["w"] = self.t_set([inp["src_w"]], dep, wdep, inp["zdt0"], "cubic", False)[0]
        out["tracers"] = self.t_set(inp["tracers"], dep, wdep, inp["zdt0"], "mono" if mono else "cubic", mono)
        return out

    def departure(self, dep, start_wp):
        wp = start_wp.clone()
        wp[:, :, 2:self.nj + 2, 2:self.ni + 2] = dep
        return wp

    def fixer(self, st, inp, dep, wdep):
        """Bounds, boundary fluxes and the fixer of weight |high - low order|."""
        H, nk = self.H, self.nk
        m, lin, mn, mx = self.t_set(inp["tracers"], dep, wdep, inp["zdt0"], "mono", False, post=True)
        core, rb = self.box("core"), self.box("b")
        own = (slice(None), slice(H, H + self.nj), slice(H, H + self.ni))
        inner = torch.zeros((self.njt, self.nit), dtype=torch.bool, device="cuda")
        inner[H:H + self.nj, H:H + self.ni][core] = True
        dom = torch.zeros_like(inner)
        dom[H:H + self.nj, H:H + self.ni] = True
        zero = torch.zeros((), device="cuda", dtype=torch.float64)
        src = inp["tracers"]
        fo = self.t_set([torch.where(inner, f, zero.to(f.dtype)) for f in src], dep, wdep, inp["zdt0"], "cubic", False,
                        box="b")
        fi = self.t_set([torch.where(dom & ~inner, f, zero.to(f.dtype)) for f in src], dep, wdep, inp["zdt0"], "cubic",
                        False, box="b")
        ap, am, area = st["air_p"].double(), st["air_m"].double(), st["mask"]
        mass = lambda f, a, box: ((f * a)[own] * area)[(slice(None),) + box].sum()  # noqa: E731
        diag = []
        for q, f in enumerate(src):
            fo[q].masked_fill_(inner, 0.0)
            fi[q].masked_fill_(dom & ~inner, 0.0)
            d = [mass(f.double(), ap, core), mass(m[q], am, core), mass(fo[q], am, rb), mass(fi[q], am, rb)]
            tot = d[0] + d[3] - d[2]
            deficit = d[1] - tot
            sign = 1.0 if float(deficit) >= 0 else -1.0
            h = m[q] - lin[q]
            w = torch.where(torch.sign(h) * sign >= 0, h.abs() * sign, torch.zeros_like(h))
            wei = mass(w, am, core)
            lam = deficit / wei
            new = m[q] - lam * w
            corr = lam * w
            new = torch.where((corr > 0) & (new < mn[q]), mn[q], new)
            new = torch.where((corr < 0) & (new > mx[q]), mx[q], new)
            bc_r = mass(new, am, core)
            new = new * (tot / bc_r)
            m[q][own][(slice(None),) + core] = new[own][(slice(None),) + core]
            diag.append(torch.stack(d + [wei, lam, bc_r, mass(m[q], am, core)]))
        return dict(tracers=m, fo=fo, fi=fi, diag=torch.stack(diag))


def exact(case, seed):
    kind = case["kind"]
    if kind == "ilmc":  # point after point in loop order: too long
        return None
    if kind == "batch":
        out = []
        for p in range(min(8, case["domains"])):
            cfg = _config(case, seed, p)
            inp = _inputs(cfg, case["prec"])
            ex = _Exact(cfg)
            wp, _ = _start(cfg, inp, case["prec"])
            dep, wdep = ex.trajectory(inp, wp[:, :, 2:cfg.nj + 2, 2:cfg.ni + 2], 2)
            f = ex.fields(inp, dep, wdep, case["mono"])
            out.append(dict(wpxyz=ex.departure(dep, wp), fields=[f["u"], f["v"], f["w"]] + f["tracers"]))
        return out
    if kind == "interp":
        s = prepare(case, seed)
        cfg = _config(case, seed)
        ex = _Exact(cfg)
        p = s["pos"].double()
        st = ex.stencil(p[:, 0], p[:, 1], p[:, 2], ex.zt)
        r = [ex.cubic(f, st, True) for f in s["ext"]]
        return {k: torch.stack([v[q] for v in r]) for q, k in enumerate(("d", "lin", "mn", "mx"))}
    cfg = _config(case, seed)
    inp = _inputs(cfg, case["prec"])
    ex = _Exact(cfg)
    if kind == "cold":  # the iteration's fixed point
        i = torch.arange(1, cfg.ni + 1, device="cuda", dtype=torch.float64)
        j = torch.arange(1, cfg.nj + 1, device="cuda", dtype=torch.float64).view(-1, 1)
        k = torch.arange(1, cfg.nk + 1, device="cuda", dtype=torch.float64).view(-1, 1, 1)
        full = (cfg.nk, cfg.nj, cfg.ni)
        start = torch.stack([i.expand(full), j.expand(full), k.expand(full)])
        dep, wdep = ex.trajectory(inp, start, 9)
        wp = torch.zeros((3, cfg.nk, cfg.nj + 4, cfg.ni + 4), device="cuda", dtype=torch.float64)
        return dict(ex.fields(inp, dep, wdep, case["mono"]), wpxyz=ex.departure(dep, wp))
    wp, px = _start(cfg, inp, case["prec"])
    start = wp[:, :, 2:cfg.nj + 2, 2:cfg.ni + 2]
    if px is not None:
        start = px.double().permute(3, 0, 1, 2).contiguous()
    dep, wdep = ex.trajectory(inp, start, 2)
    if kind == "qv":
        r = ex.t_set(inp["tracers"], dep, wdep, inp["zdt0"], "qv", True, post=True)
        return dict(zip(("tracers", "lin", "mn", "mx"), r))
    if kind == "fixer":
        return ex.fixer(prepare(case, seed), inp, dep, wdep)
    out = dict(ex.fields(inp, dep, wdep, case["mono"]), wpxyz=ex.departure(dep, wp))
    if px is not None:
        x, y = ex.clip(dep[0], dep[1])
        out["pxyzm"] = torch.stack([x, y, dep[2]], dim=-1)
    return out
