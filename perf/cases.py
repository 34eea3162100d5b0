"""The work whose speed this framework is judged by: the dynamics step and its routines.

A forecast calls `DycoreState.step` once a time step (the state stays on the
device); a host model that keeps its own time loop calls the routines of the
step one by one through `Dycore` on arrays it owns, in the reference's argument
order.  Both are here, from the smallest served request (glvl 5, nvl 38) to a
global forecast at glvl 8, in FP32-mixed precision (production) and in FP64
(the plain configuration).

Inputs are a balanced, noisy state made from the seed alone: by the library's
own state generator for the step (what the serving loop does), by torch in FP64
for the routines.  `exact` evaluates the routines in plain torch FP64 from
their definitions.
"""
import functools
import math

import numpy as np
import torch

import fimocn_subx_realtime_hera_apr2020_gb300 as F

CP, RD, P1000, GRAV = 1004.6855, 287.0586, 100000.0, 9.80665
OMEGX2, EARTH, PI = 1.4584e-4, 6371220.0, 3.14159265
PTOP, SIGMA_PS, NOISE = 30.0, 200.0, 1.0
F64 = torch.float64

# what a driver keeps of a step: the prognostic state, the AB3 histories, the
# mass fluxes; a single forecast also the diagnostics
STATE = ["us3d", "vs3d", "dp3d", "pr3d", "ex3d", "ph3d", "mp3d", "tr3d", "trdp", "u_tdcy", "v_tdcy", "dp_tdcy",
         "dpl_tdcy", "trc_tdcy", "trl_tdcy", "massfx"]
DIAG = ["ws3d", "sdot", "relvor", "psrf", "ptdcy"]


def listed():
    def step(name, glvl, nvl, ntra, prec="f32", members=1):
        return dict(name=name, kind="step", glvl=glvl, nvl=nvl, ntra=ntra, prec=prec, members=members)

    def routine(kind, glvl, nvl, ntra, prec="f32"):
        return dict(name="%s_g%d_l%d_t%d_%s" % (kind, glvl, nvl, ntra, prec), kind=kind, glvl=glvl, nvl=nvl,
                    ntra=ntra, prec=prec, members=1)

    return [
        # one time step of the smallest served request: launches and latency
        step("step_g5_l38_t5_f32", 5, 38, 5),
        # a small ensemble advanced as one batch
        step("step_g6_l64_t11_x4_f32", 6, 64, 11, members=4),
        # the largest served request: 20 tracers and theta
        step("step_g7_l64_t21_f32", 7, 64, 21),
        # a global forecast at the finest grid of the benchmark
        step("step_g8_l64_t11_f32", 8, 64, 11),
        # the plain FP64 forecast of the accuracy runs
        step("step_g6_l64_t11_f64", 6, 64, 11, prec="f64"),
        # a host model's own time loop, routine by routine, on its arrays
        routine("edges", 7, 64, 11),
        routine("cnuity", 7, 64, 5),
        routine("trcadv", 7, 64, 11),
        routine("momtum", 7, 64, 5),
        routine("column", 7, 64, 11),
        # the same loop in FP64 at the size of the plain configuration, and
        # with a column height that is no multiple of a vector
        routine("trcadv", 5, 37, 5, "f64"),
        routine("column", 5, 38, 5, "f64"),
    ]


def draw(rng):
    """glvl 5..8, 26..64 layers (odd ones among them), 5..21 tracers."""
    kind = rng.choice(["step", "step", "step", "edges", "cnuity", "trcadv", "momtum", "column"])
    prec = "f64" if rng.random() < 0.25 else "f32"
    nvl = rng.choice([38, 64, int(round(math.exp(rng.uniform(math.log(26), math.log(64)))))])
    ntra = int(round(math.exp(rng.uniform(math.log(5), math.log(21)))))
    top = 6 if prec == "f64" else 8 if kind == "step" else 7
    glvl = rng.randint(5, top)
    members = 1
    if glvl == 8:
        ntra = min(ntra, 11)
    elif kind == "step" and glvl <= 6:
        members = rng.choice([1, 1, 2, 3, 4])
    if prec == "f64" and glvl == 6:
        ntra, members = min(ntra, 11), 1
    return dict(kind=kind, glvl=glvl, nvl=nvl, ntra=ntra, prec=prec, members=members)


# ---- grid tables and configuration -----------------------------------------
def _config(case):
    nvl = case["nvl"]
    if nvl in (38, 64):
        thetac, dpsig = F.vertical_tables(nvl)
    else:  # a caller's own levels: the 64-layer tables resampled
        th, dp = F.vertical_tables(64)
        at = np.linspace(0.0, 63.0, nvl)
        thetac = np.interp(at, np.arange(64.0), th)
        dpsig = np.interp(at, np.arange(64.0), dp)
        dpsig = dpsig * (dp.sum() / dpsig.sum())
    # half of the grid's default time step: stays stable without physics
    return F.FimConfig(nvl=nvl, ntra=case["ntra"], dt=0.5 * F.default_dt(case["glvl"]), precision=case["prec"],
                       members=case["members"], thetac=thetac, dpsig=dpsig)


class Tables:
    """Grid tables of one level as FP64 torch tensors (0-based indices)."""

    def __init__(self, glvl):
        g = F.Grid.cached(glvl)
        n = g.nip

        def dev(a, *shape):
            return torch.as_tensor(np.ascontiguousarray(a), device="cuda").reshape(n, *shape)

        self.n = n
        self.np = dev(g.nprox).long()
        self.prox = dev(g.prox, 6).long() - 1
        self.live = torch.arange(6, device="cuda")[None, :] < self.np[:, None]
        self.proxs = torch.where(self.live, dev(g.proxs, 6).long() - 1, 0)
        self.cs, self.sn = dev(g.cs, 6, 4), dev(g.sn, 6, 4)
        self.svc, self.sve = dev(g.sidevec_c, 6, 2), dev(g.sidevec_e, 6, 2)
        self.sideln, self.hf = dev(g.sideln, 6), dev(g.hfcoef, 6, 6)
        self.lat, self.area = dev(g.lat), dev(g.area)
        self.rarea = 1.0 / self.area
        self.corio = OMEGX2 * torch.sin(self.lat)
        self.grnd = EARTH * 2.0 * PI * torch.cos(self.lat) / 86164.0
        e = torch.arange(6, device="cuda")[None, :]
        row = torch.arange(n, device="cuda")[:, None]
        self.trail = self.prox[row, (e - 1) % self.np[:, None]]
        self.lead = self.prox[row, (e + 1) % self.np[:, None]]


@functools.lru_cache(maxsize=4)
def _tables(glvl):
    return Tables(glvl)


# ---- the routines in plain FP64 torch; cell fields (n, L), edges (n, 6, L) --
def _edge_winds(t, f):
    """edgvar1: four-cell interpolation to the edges in the edge's own frame."""
    n, L = f["u"].shape
    out = {k: torch.zeros(n, 6, L, dtype=F64, device="cuda") for k in ("u", "v", "lp", "mont", "uvsq", "th")}
    play = f["pres"][:, :L] + f["pres"][:, 1:]
    th = f["tr"][0]
    me = torch.arange(n, device="cuda")
    for e in range(6):
        cells = (me, t.prox[:, e], t.trail[:, e], t.lead[:, e])
        wgt = (2.0, 2.0, 1.0, 1.0)
        ue, ve, mag, lp, mo, te = 0.0, 0.0, 0.0, 0.0, 0.0, 0.0
        for q, (x, w) in enumerate(zip(cells, wgt)):
            c, s = t.cs[:, e, q, None], t.sn[:, e, q, None]
            a, b = c * f["u"][x] + s * f["v"][x], -s * f["u"][x] + c * f["v"][x]
            ue, ve, mag = ue + w * a, ve + w * b, mag + w * torch.sqrt(a * a + b * b)
            lp = lp + 0.5 * w * play[x]
            mo, te = mo + w * f["mont"][x], te + w * th[x]
        ue, ve, mag = ue / 6.0, ve / 6.0, mag / 6.0
        q = mag / torch.clamp(torch.sqrt(ue * ue + ve * ve), min=0.001)
        ue, ve = ue * q, ve * q
        live = t.live[:, e, None]
        for k, x in (("u", ue), ("v", ve), ("lp", lp / 6.0), ("mont", mo / 6.0),
                     ("uvsq", 0.5 * (ue * ue + ve * ve)), ("th", te / 6.0)):
            out[k][:, e] = torch.where(live, x, 0.0)
    return out


def _edge_fit(t, x):
    """edgvar3: least-squares edge values of both cells of an edge, averaged."""
    n, L = x.shape
    own = torch.zeros(n, 6, L, dtype=F64, device="cuda")
    d = torch.where(t.live[:, :, None], x[t.prox] - x[:, None], 0.0)
    for e in range(6):
        own[:, e] = torch.where(t.live[:, e, None], x + (d * t.hf[:, e, :, None]).sum(1), 0.0)
    return torch.where(t.live[:, :, None], 0.5 * (own + own[t.prox, t.proxs]), 0.0)


def _limit(t, cell, low, old, anti, ab, thick):
    """Zalesak limiters of the antidiffusive fluxes; cell bounds over the 1-ring."""
    ab1, ab2, ab3 = ab
    out, inn = torch.clamp(anti, min=0.0).sum(1), torch.clamp(-anti, min=0.0).sum(1)
    both = torch.stack((torch.maximum(cell, low), torch.minimum(cell, low)))
    mx = torch.maximum(both[0], both[0][t.prox].amax(1)).clamp(min=0.0)
    mn = torch.minimum(both[1], both[1][t.prox].amin(1)).clamp(min=0.0)
    o, v = old
    ar = t.area[:, None] / ab1
    qp = ((mx - low) * thick - (ab2 * o.clamp(max=0.0) + ab3 * v.clamp(min=0.0))) * ar
    qm = ((low - mn) * thick + (ab2 * o.clamp(min=0.0) + ab3 * v.clamp(max=0.0))) * ar
    rp = (qp / inn.clamp(min=1e-11)).clamp(0.0, 1.0)
    rm = (qm / out.clamp(min=1e-11)).clamp(0.0, 1.0)
    clip = torch.where(anti >= 0, torch.minimum(rm[:, None], rp[t.prox]), torch.minimum(rp[:, None], rm[t.prox]))
    return anti * clip, mx, mn


def _continuity(t, f, ue, ve, dpe, lpe, slots, ab, dt):
    """cnuity: f has u, v, dp, pres; slots = (dp_of, dp_vof, dplo_of, dplo_vof)."""
    live = t.live[:, :, None]
    vn = torch.where(live, t.sve[:, :, 1:2] * ue - t.sve[:, :, 0:1] * ve, 0.0)
    vx = vn[t.prox, t.proxs]
    dp = f["dp"]
    low = torch.where(live, 0.5 * ((vn + vn.abs()) * dp[:, None] - (vx + vx.abs()) * dp[t.prox]), 0.0)
    anti = torch.where(live, vn * dpe - low, 0.0)
    del vn, vx
    ab1, ab2, ab3 = ab
    tlo = -low.sum(1) * t.rarea[:, None]
    dplo = dp + ab1 * tlo + ab2 * slots[2] + ab3 * slots[3]
    anti, _, _ = _limit(t, dp, dplo, slots[:2], anti, ab, 1.0)
    tdp = tlo - anti.sum(1) * t.rarea[:, None]
    rate = ab1 * tdp + ab2 * slots[0] + ab3 * slots[1]
    new = dp + rate
    pres = f["pres"].clone()
    pres[:, :-1] = pres[:, -1:] + new.flip(1).cumsum(1).flip(1)
    lyr = rate / dt
    above = lyr.flip(1).cumsum(1).flip(1) - lyr
    gx = torch.where(live, lpe * t.svc[:, :, 1:2], 0.0).sum(1)
    gy = -torch.where(live, lpe * t.svc[:, :, 0:1], 0.0).sum(1)
    omega = above + 0.5 * lyr + (f["u"] * gx + f["v"] * gy) * t.rarea[:, None]
    return dict(dp=new, pres=pres, exner=CP * (pres / P1000) ** (RD / CP), tdp=tdp, tlo=tlo, flux=low + anti,
                omega=omega)


def _tracer(t, x, xdp, edge, flux, dp, slots, ab):
    """trcadv of one tracer; slots = (tdcy_of, tdcy_vof, low_of, low_vof)."""
    live = t.live[:, :, None]
    fx = flux[t.prox, t.proxs]
    low = torch.where(live, 0.5 * ((flux + flux.abs()) * x[:, None] - (fx + fx.abs()) * x[t.prox]), 0.0)
    anti = torch.where(live, flux * edge - low, 0.0)
    del fx
    ab1, ab2, ab3 = ab
    tlo = -low.sum(1) * t.rarea[:, None]
    del low
    mx = torch.maximum(x, x[t.prox].amax(1)).clamp(min=0.0)
    mn = torch.minimum(x, x[t.prox].amin(1)).clamp(min=0.0)
    thick = dp.clamp(min=1e-11)
    xlo = torch.maximum(mn, torch.minimum(mx, (xdp + ab1 * tlo + ab2 * slots[2] + ab3 * slots[3]) / thick))
    anti, mx, mn = _limit(t, x, xlo, slots[:2], anti, ab, dp)
    tx = tlo - anti.sum(1) * t.rarea[:, None]
    new = xdp + ab1 * tx + ab2 * slots[0] + ab3 * slots[1]
    return torch.maximum(mn, torch.minimum(mx, new / thick)), new, tx, tlo


def _momentum(t, cfg, f, w, slots, ab):
    """momtum: dissipation, pressure gradient, vorticity, AB3, Rayleigh damping."""
    n, L = f["u"].shape
    k = torch.arange(1, L + 1, dtype=F64, device="cuda")
    nd = int(0.1 * L)
    wgt = ((k - L + nd) / nd).clamp(min=0.0)
    dfl = cfg.dt * (cfg.veldff_bkgnd * (1.0 - wgt) + max(cfg.veldff_bkgnd, cfg.veldff_boost) * wgt)
    u, v, dp = f["u"], f["v"], f["dp"].clamp(min=1e-11)
    wu = u + t.grnd[:, None]
    du, dv = torch.zeros_like(u), torch.zeros_like(v)
    for e in range(6):
        x, live = t.prox[:, e], t.live[:, e, None]
        c0, s0, c1, s1 = (a[:, e, q, None] for a, q in ((t.cs, 0), (t.sn, 0), (t.cs, 1), (t.sn, 1)))
        jump_u = (c1 * wu[x] + s1 * v[x]) - (c0 * wu + s0 * v)
        jump_v = (-s1 * wu[x] + c1 * v[x]) - (-s0 * wu + c0 * v)
        h = dfl * t.sideln[:, e, None] * 2.0 * (dp * dp[x] / (dp + dp[x])) * t.rarea[:, None] / dp
        du += torch.where(live, (c0 * jump_u - s0 * jump_v) * h, 0.0)
        dv += torch.where(live, (s0 * jump_u + c0 * jump_v) * h, 0.0)
    u, v = u + du, v + dv
    exm = 0.5 * (f["exner"][:, :L] + f["exner"][:, 1:])
    pot = w["mont"] + w["uvsq"] - exm[:, None] * w["th"]
    live = t.live[:, :, None]
    r = t.rarea[:, None]
    gx = -torch.where(live, pot * t.svc[:, :, 1:2], 0.0).sum(1) * r
    gy = torch.where(live, pot * t.svc[:, :, 0:1], 0.0).sum(1) * r
    rv = torch.where(live, t.sve[:, :, 0:1] * w["u"] + t.sve[:, :, 1:2] * w["v"], 0.0).sum(1) * r
    ut, vt = gx + (t.corio[:, None] + rv) * v, gy - (t.corio[:, None] + rv) * u
    u = u + ab[0] * ut + ab[1] * slots[0] + ab[2] * slots[1]
    v = v + ab[0] * vt + ab[1] * slots[2] + ab[2] * slots[3]
    q = (u[:, -3:] ** 2 + v[:, -3:] ** 2).amax(1) / cfg.rlthresh ** 2
    q = torch.where(q > 1.0, torch.sqrt((q - 1.0).clamp(min=0.0) * q), 0.0)
    fac = torch.where(k >= L - int(0.25 * L), cfg.rleigh * 2.0 ** (cfg.rltaper * (k - L)) * cfg.dt / 86400.0, 0.0)
    damp = 1.0 - q[:, None] * fac
    return u * damp, v * damp, rv, ut, vt


def _hydrostatic(ex, th, ph0):
    """hystat: Montgomery potential and geopotential of the columns."""
    L = th.shape[1]
    mont = (ex[:, 0] * th[:, 0] + ph0)[:, None].expand_as(th).clone()
    mont[:, 1:] += (ex[:, 1:L] * (th[:, 1:] - th[:, :-1])).cumsum(1)
    ph = torch.empty_like(ex)
    ph[:, 0] = ph0
    ph[:, 1:] = mont - th * ex[:, 1:]
    return mont, ph


def _inflate(cfg, p0, ex):
    """Minimum layer thicknesses, bottom up, then near the top; ex is a list of (n)."""
    L = len(ex) - 1
    thin = RD / P1000

    def cushion(a, b):
        m = torch.minimum(a, 2.0 * b)
        return 0.25 * m * m / b + torch.maximum(a, 2.0 * b) - b

    extop = CP * (cfg.ptop / P1000) ** (RD / CP)
    shrink = ((p0 / P1000 - 0.2) / 0.8).clamp(max=1.0)
    total = torch.zeros_like(p0)
    last = torch.ones_like(p0)
    for k in range(1, L):
        dp0 = RD * float(cfg.dpsig[k - 1]) / P1000 * shrink
        total = total + dp0
        if k <= cfg.kbl:
            last = torch.full_like(p0, k + 1.0)
            ex[k] = ex[k - 1] - dp0
            continue
        soft = (dp0 / torch.clamp(1.25 * 2.0 ** (k - last), max=10.0)).clamp(min=RD * 100.0 / P1000)
        dp0 = torch.where(k > last, soft, dp0)
        dp1 = cushion((ex[k - 1] - torch.minimum(ex[k], ex[0] - total)).clamp(min=0.0), dp0)
        hit = ex[k - 1] - dp1 < ex[k] - thin
        last = torch.where(hit & (last == k), k + 1.0, last)
        ex[k] = torch.where(hit, (ex[k - 1] - dp1).clamp(min=extop), ex[k])
    going = torch.full(p0.shape, cfg.thktop > 0.0, device="cuda")
    for k in range(L, 1, -1):
        q = (ex[k - 1] / CP) ** 2.5
        dp0 = RD * cfg.thktop / P1000 / (1.0 + (0.25 * (L - k)) ** 2) / q
        dp1 = cushion((ex[k - 1] - ex[k]).clamp(min=0.0), dp0)
        ex[k - 1] = torch.where(going & (ex[k] + dp1 > ex[k - 1] + thin), ex[k] + dp1, ex[k - 1])
        going = going & ~(ex[k - 1] < ex[k - 2] - dp0)


def _restore(tg, th, ex):
    """restp_1d: the interfaces that give the target theta column the old one's integral."""
    L = len(th)
    old = list(th)
    for k in range(L - 1, 0, -1):
        old[k - 1] = torch.minimum(old[k], old[k - 1])
    # a layer at theta spans the target interval it is clamped to: the new
    # interface between k and k+1 is the Exner function averaged over theta
    n = [torch.full_like(ex[0], float(x)) for x in tg]
    n[0] = torch.minimum(torch.minimum(old[0], old[-1]), n[0])
    n[-1] = torch.maximum(torch.maximum(old[0], old[-1]), n[-1])
    old, ex_ = torch.stack(old), torch.stack(ex)
    new = [ex[0]]
    for k in range(L - 1):
        lo, hi = n[k], n[k + 1]
        c = torch.minimum(hi, torch.maximum(lo, old))                      # (L, n)
        steps = torch.cat((c[:1] - lo, c[1:] - c[:-1], hi[None] - c[-1:]))  # below, between, above
        mean = (ex_ * steps).sum(0) / torch.where(hi > lo, hi - lo, 1.0)
        new.append(torch.where(hi > lo, mean, new[k]))
    new.append(ex[L])
    return new


def _regrid(cfg, its, th, ex, p0):
    """regrid_1d: th (n, L), ex (n, L+1) -> new interface Exner function, list of (n)."""
    L = th.shape[1]
    tg = cfg.thetac
    thin, tol = RD / P1000, 0.001
    ex = [ex[:, k].clone() for k in range(L + 1)]
    th = [th[:, k].clone() for k in range(L)]
    for k in range(L):
        ex[k + 1] = torch.where(ex[k] < ex[k + 1] - thin, ex[k], ex[k + 1])
    for k in range(L - 2, -1, -1):
        th[k] = torch.minimum(th[k], th[k + 1])
    top = float(tg[-1])
    going = torch.ones_like(p0, dtype=torch.bool)
    for k in range(L, 1, -1):
        going = going & ~(th[k - 1] <= top + tol)
        if not bool(going.any()):
            break
        w1, w2 = (ex[k - 2] - ex[k - 1]).clamp(min=0.0), (ex[k - 1] - ex[k]).clamp(min=thin)
        mix = (th[k - 2] * w1 + th[k - 1] * w2) / (w1 + w2)
        merge = going & (mix > top - tol)
        split = going & ~merge
        gap = top - th[k - 2]
        moved = (ex[k - 1] * (th[k - 1] - th[k - 2]) + ex[k] * (top - th[k - 1])) / torch.where(split, gap, 1.0)
        moved = torch.minimum(ex[k - 2], torch.maximum(ex[k], moved))
        ex[k - 1] = torch.where(merge, ex[L], torch.where(split, moved, ex[k - 1]))
        for j in range(k - 2, L):
            x = torch.where(merge, mix, th[j])
            th[j] = torch.where(split, top, x) if j >= k - 1 else x
        going = merge
    new = _restore(tg, th, ex)
    act = torch.ones_like(p0, dtype=torch.bool)
    for _ in range(3):  # heat diffusion, until no column has an interface out of order
        src, out = list(new), list(new)
        heat = [torch.zeros_like(p0) for _ in range(L)]
        for j in range(1, L - 1):
            cnv = GRAV / float(tg[j])
            h = 0.1 * cnv * cnv * 0.5 * float(tg[j + 1] - tg[j - 1]) / (src[j] - src[j + 1]).clamp(min=0.03 * cnv)
            heat[j] = torch.where((src[j] < src[0] - 0.01) & (src[j + 1] > src[L] + 0.01), h, 0.0)
        for k in range(1, L):
            x = src[k] + (heat[k] - heat[k - 1]) / float(tg[k] - tg[k - 1])
            x = torch.maximum(src[k + 1], torch.minimum(src[k - 1], x))
            out[k] = torch.where((src[k] < src[0] - 0.01) & (src[k] > src[L] + 0.01) & act, x, src[k])
        new = out
        event = torch.zeros_like(act)
        for k in range(1, L + 1):
            event |= new[k] > new[k - 1] + thin
        act = act & event
        if not bool(act.any()):
            break
    # equilb: thickness differences of neighbouring layers evened out
    slak = 0.1 * its / (10.0 + its)
    for k in range(3, L - 1):
        d = [new[k + q] - new[k + q + 1] for q in range(-3, 2)]
        goal = 0.5 * (d[2] + torch.minimum(d[1], d[3]))
        do = ~(new[k - 3] > new[0] - thin) & (d[1] > d[0]) & (d[3] > d[4]) & (d[1] > goal) & (d[3] > goal)
        a = torch.minimum(d[1] - goal, goal - d[2]) * slak
        b = torch.minimum(d[3] - goal, goal - d[2]) * slak
        t2, t3, t4 = (float(x) for x in tg[k - 2:k + 1])
        if t3 > t2 and t4 > t3:
            ratio = (t4 - t3) / (t3 - t2)
            a, b = (a, a / ratio) if ratio > 1.0 else (b * ratio, b)
        new[k - 1] = torch.where(do, new[k - 1] + a, new[k - 1])
        new[k] = torch.where(do, new[k] - b, new[k])
    _inflate(cfg, p0, new)
    return new


def _remap(xo, xn, y):
    """pcwise with PLM and one-layer migration; xo, xn (n, L+1) decreasing, y (n, L)."""
    small = 1e-22
    fo, fn = (xo[:, :-1] - xo[:, 1:]).clamp(min=0.0), (xn[:, :-1] - xn[:, 1:]).clamp(min=0.0)
    L = y.shape[1]
    y = list(y.unbind(1))
    for k in range(L - 2, -1, -1):
        y[k] = (y[k] * fo[:, k] + y[k + 1] * small) / (fo[:, k] + small)
    for k in range(1, L):
        y[k] = (y[k] * fo[:, k] + y[k - 1] * small) / (fo[:, k] + small)
    y = torch.stack(y, 1)
    m, c, p = y[:, :-2], y[:, 1:-1], y[:, 2:]
    s = torch.where((p - m) * (m + p - 2.0 * c) > 0.0, c - m, p - c)
    s = torch.where((c <= torch.minimum(m, p)) | (c >= torch.maximum(m, p)), 0.0, s)
    slope = torch.zeros_like(y)
    slope[:, 1:-1] = s
    dz = xo[:, 1:-1] - xn[:, 1:-1]  # interfaces between layers, upward positive
    up = dz > 0.0
    thick = torch.where(up, fo[:, 1:], fo[:, :-1])
    slab = torch.minimum(thick, dz.abs())
    x = slab / torch.where(thick > 0.0, thick, 1.0)
    val = torch.where(up, y[:, 1:] + slope[:, 1:] * 0.5 * (x - 1.0), y[:, :-1] + slope[:, :-1] * 0.5 * (1.0 - x))
    flux = torch.zeros_like(xo)
    flux[:, 1:-1] = torch.where(slab > 0.0, -dz * val, 0.0)
    return (y * fo - (flux[:, 1:] - flux[:, :-1]) + y * small) / (fn + small)


def _hybrid(t, cfg, its, f):
    """hybgen: f has u, v, tr (T, n, L), exner, pres; returns the new column state."""
    ex, pr, tr = f["exner"], f["pres"], f["tr"]
    L = ex.shape[1] - 1
    new = torch.stack(_regrid(cfg, its, tr[0], ex, pr[:, 0]), 1)
    k = torch.arange(1, L + 2, dtype=F64, device="cuda")
    d1, d2 = (cfg.kbl + 1) - k, (L + 1) - k
    smoo = cfg.dt * cfg.intfc_smooth * (d1 * d1 / (9.0 + d1 * d1)) * (d2 * d2 / (9.0 + d2 * d2))
    smoo = torch.where((k >= cfg.kbl + 2) & (k <= L), smoo, 0.0)
    div = torch.zeros_like(new)
    for e in range(6):
        div += torch.where(t.live[:, e, None], (new - new[t.prox[:, e]]) * t.sideln[:, e, None], 0.0)
    new = list((new - div * smoo * t.rarea[:, None]).unbind(1))
    _inflate(cfg, pr[:, 0], new)
    new = torch.stack(new, 1)
    if its > 0:
        new = cfg.slak * new + (1.0 - cfg.slak) * ex
    lo, hi = 0.0001 * ex[:, 1:-1] + 0.9999 * ex[:, 2:], 0.0001 * ex[:, 1:-1] + 0.9999 * ex[:, :-2]
    new[:, 1:-1] = torch.maximum(lo, torch.minimum(hi, new[:, 1:-1]))
    prn = P1000 * (new / CP) ** (CP / RD)
    dp = prn[:, :-1] - prn[:, 1:]
    pk, pkn = ex * pr / CP, new * prn / CP
    for a, b in ((prn, pr), (pkn, pk)):
        a[:, 0], a[:, L] = b[:, 0], b[:, L]
    out = [None] + [_remap(pr, prn, x) for x in tr[1:]]
    th = list(_remap(pk, pkn, tr[0]).unbind(1))
    w = (pkn[:, :-1] - pkn[:, 1:]).clamp(min=0.0)
    w = torch.maximum(w, pkn[:, :1] * 1e-6)
    for k in range(L - 1, 1, -1):
        a, b = (th[k - 1] - float(cfg.thetac[k - 1])) * w[:, k - 1], (th[k] - float(cfg.thetac[k])) * w[:, k]
        x = torch.where((b > 0) & (a < 0), torch.minimum(b, -a), torch.where((b < 0) & (a > 0), -torch.minimum(a, -b), 0.0))
        th[k - 1], th[k] = th[k - 1] + x / w[:, k - 1], th[k] - x / w[:, k]
    out[0] = torch.stack(th, 1)
    exn = new.cummin(1)[0]
    return dict(u=_remap(pr, prn, f["u"]), v=_remap(pr, prn, f["v"]), tr=out, sdot=exn - ex, exner=exn, dp=dp, pres=prn)


# ---- inputs ------------------------------------------------------------------
def _balanced(t, cfg, seed):
    """A noisy balanced state, FP64: u, v, dp, pres, exner, tr (T, n, L), mont."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    n, L, T = t.n, cfg.nvl, cfg.ntra

    def normal(*s):
        return torch.randn(*s, generator=gen, device="cuda", dtype=F64)

    ps = P1000 + SIGMA_PS * normal(n)
    share = torch.as_tensor(cfg.dpsig / cfg.dpsig.sum(), device="cuda")
    dp = (ps - PTOP)[:, None] * share
    pres = torch.full((n, L + 1), PTOP, dtype=F64, device="cuda")
    pres[:, :L] += dp.flip(1).cumsum(1).flip(1)
    ex = CP * (pres / P1000) ** (RD / CP)
    u = 35.0 * torch.cos(t.lat)[:, None] + NOISE * normal(n, L)
    v = NOISE * normal(n, L)
    tr = torch.rand(T, n, L, generator=gen, device="cuda", dtype=F64) * 1e-2
    tr[0] = torch.linspace(300.0, 600.0, L, dtype=F64, device="cuda") + 0.2 * normal(n, L)
    mont, _ = _hydrostatic(ex, tr[0], torch.zeros(n, dtype=F64, device="cuda"))
    return dict(u=u, v=v, dp=pres[:, :L] - pres[:, 1:], pres=pres, exner=ex, tr=tr, mont=mont), gen


def _history(gen, now, slots=(1, 2)):
    """Three AB3 slots of a tendency: the two old ones near `now`, slot 0 (rewritten) zero."""
    out = torch.zeros(3, *now.shape, dtype=F64, device="cuda")
    for s in slots:
        out[s] = now * (1.0 + 0.1 * torch.randn(now.shape, generator=gen, device="cuda", dtype=F64))
    return out


def _ab3(dt):
    return (dt * 23.0 / 12.0, -dt * 16.0 / 12.0, dt * 5.0 / 12.0)


ITS = 4  # the routines' first pass: AB3 in full swing; slots nf, of, vof = 0, 2, 1 then


def _inputs(case, seed):
    """The arrays a host model holds when it calls the routine, in its precision."""
    t, cfg = _tables(case["glvl"]), _config(case)
    f, gen = _balanced(t, cfg, seed)
    n, L, T = t.n, cfg.nvl, cfg.ntra
    kind, euler = case["kind"], (cfg.dt, 0.0, 0.0)
    zero = torch.zeros(n, L, dtype=F64, device="cuda")
    a = dict(u=f["u"], v=f["v"], dp=f["dp"], pres=f["pres"], exner=f["exner"], mont=f["mont"], tr=f["tr"])
    if kind in ("cnuity", "trcadv", "momtum"):
        w = _edge_winds(t, f)
    if kind in ("cnuity", "trcadv"):
        a.update(ue=w["u"], ve=w["v"], lpe=w["lp"], dpe=_edge_fit(t, f["dp"]))
        c = _continuity(t, f, a["ue"], a["ve"], a["dpe"], a["lpe"], (zero,) * 4, euler, cfg.dt)
        a.update(tdp=_history(gen, c["tdp"]), tlo=_history(gen, c["tlo"]))
    if kind == "trcadv":
        flux = c["flux"].expand(3, n, 6, L).contiguous()
        te, tt, tl = [], [], []
        for q in range(T):
            te.append(w["th"] if q == 0 else _edge_fit(t, f["tr"][q]))
            _, _, x, lo = _tracer(t, f["tr"][q], f["tr"][q] * f["dp"], te[-1], flux[0], c["dp"], (zero,) * 4, euler)
            tt.append(_history(gen, x))
            tl.append(_history(gen, lo))
        a = dict(te=torch.stack(te), tr=f["tr"], trdp=f["tr"] * f["dp"], tt=torch.stack(tt), tl=torch.stack(tl),
                 flux=flux, dp=c["dp"])
    if kind == "cnuity":
        a["flux"] = torch.zeros(3, n, 6, L, dtype=F64, device="cuda")
        del a["tr"], a["mont"]
    if kind == "momtum":
        _, _, _, ut, vt = _momentum(t, cfg, f, w, (zero,) * 4, euler)
        a.update(ue=w["u"], ve=w["v"], the=w["th"], monte=w["mont"], uvsqe=w["uvsq"], ut=_history(gen, ut),
                 vt=_history(gen, vt))
        del a["tr"], a["mont"], a["pres"]
    if kind == "column":
        # the surface pressure of the step before
        a["psrf"] = f["pres"][:, 0] - PTOP + 20.0 * torch.randn(n, generator=gen, device="cuda", dtype=F64)
        del a["mont"]
    dt = torch.float64 if case["prec"] == "f64" else torch.float32
    return {k: x.to(dt).contiguous() for k, x in a.items()}


def prepare(case, seed):
    cfg = _config(case)
    dyc = F.Dycore(F.Grid.cached(case["glvl"]), cfg)
    if case["kind"] == "step":
        st = dyc.state()
        for m in range(cfg.members):
            st.synthetic(m, 1000 * int(seed) + m, cfg.ntra, sigma_ps=SIGMA_PS, noise=NOISE)
        st.init()
        names = STATE + (DIAG if cfg.members == 1 else [])
        # views of the state's own buffers; each keeps the state that owns them
        views = {"%s_%d" % (n, m): st.tensor(n, m) for m in range(cfg.members) for n in names}
        for x in views.values():
            x.owner = (dyc, st)
        return dict(kind="step", dyc=dyc, state=st, out=views)
    a = _inputs(case, seed)
    n, L, T = dyc.N, dyc.L, dyc.T

    def room(*shape):
        return torch.zeros(*shape, dtype=torch.float64 if case["prec"] == "f64" else torch.float32, device="cuda")

    kind = case["kind"]
    if kind == "edges":
        a.update({k: room(n, 6, L) for k in ("ue", "ve", "dpe", "lpe", "phe", "monte", "uvsqe")})
        a.update(ph=room(n, L + 1), te=room(T, n, 6, L))
    elif kind == "cnuity":
        a["omega"] = room(n, L)
    elif kind == "momtum":
        a.update(relvor=room(n, L), phe=room(n, 6, L))
    elif kind == "column":
        a.update(sdot=room(n, L + 1), ph=room(n, L + 1), mont=room(n, L), trdp=room(T, n, L), ptdcy=room(2, n))
    dyc.set_ab(3, 2, 1, *_ab3(cfg.dt))  # the first pass's abstart moves on to slots 1, 3, 2
    return dict(kind=kind, dyc=dyc, a=a, its=ITS)


def run(state):
    dyc, kind = state["dyc"], state["kind"]
    if kind == "step":
        state["state"].step(use_graph=True)
        return state["out"]
    a, its = state["a"], state["its"]
    state["its"] = its + 1
    if kind == "edges":
        args = [a[k] for k in ("u", "v", "dp", "pres", "exner", "ph", "mont", "tr", "ue", "ve", "dpe", "lpe", "phe",
                               "monte", "uvsqe", "te")]
        dyc.edgvar1(its, *args)
        dyc.edgvar3(its, *args)
        return {k: a[k] for k in ("ue", "ve", "dpe", "lpe", "monte", "uvsqe", "te")}
    dyc.abstart(its)
    if kind == "cnuity":
        dyc.cnuity(its, *[a[k] for k in ("u", "v", "ue", "ve", "dpe", "lpe", "dp", "pres", "exner", "tdp", "tlo",
                                         "flux", "omega")])
        return {k: a[k] for k in ("dp", "pres", "exner", "tdp", "tlo", "flux", "omega")}
    if kind == "trcadv":
        dyc.trcadv(its, *[a[k] for k in ("te", "tr", "trdp", "tt", "tl", "flux", "dp")])
        return {k: a[k] for k in ("tr", "trdp", "tt", "tl")}
    if kind == "momtum":
        dyc.momtum(its, *[a[k] for k in ("u", "v", "exner", "relvor", "ue", "ve", "the", "phe", "monte", "uvsqe",
                                         "ut", "vt", "dp")])
        return {k: a[k] for k in ("u", "v", "relvor", "ut", "vt")}
    # the column adjustment that opens a step, and the budgets of its result
    dyc.hybgen(its, None, *[a[k] for k in ("u", "v", "tr", "sdot", "exner", "dp", "pres")])
    dyc.hystat(its, *[a[k] for k in ("ph", "exner", "mont", "dp", "tr", "trdp", "psrf", "ptdcy")])
    qtrcr, b = dyc.globsum(its, *[a[k] for k in ("dp", "tr", "pres", "exner")])
    out = {k: a[k] for k in ("u", "v", "tr", "sdot", "exner", "dp", "pres", "ph", "mont", "trdp", "psrf", "ptdcy")}
    out.update(qtrcr=qtrcr, qmass=b["qmass"])
    return out


def exact(case, seed):
    """The routines' first pass in FP64; none for whole steps (the start-up adjustment and all routines chained)."""
    if case["kind"] == "step":
        return None
    t, cfg = _tables(case["glvl"]), _config(case)
    a = {k: x.to(F64) for k, x in _inputs(case, seed).items()}
    kind, ab = case["kind"], _ab3(cfg.dt)
    if kind == "edges":
        w = _edge_winds(t, a)
        te = torch.stack([w["th"]] + [_edge_fit(t, a["tr"][q]) for q in range(1, cfg.ntra)])
        return dict(ue=w["u"], ve=w["v"], dpe=_edge_fit(t, a["dp"]), lpe=w["lp"], monte=w["mont"], uvsqe=w["uvsq"], te=te)
    if kind == "cnuity":
        slots = (a["tdp"][2], a["tdp"][1], a["tlo"][2], a["tlo"][1])
        c = _continuity(t, a, a["ue"], a["ve"], a["dpe"], a["lpe"], slots, ab, cfg.dt)
        a["tdp"][0], a["tlo"][0], a["flux"][0] = c["tdp"], c["tlo"], c["flux"]
        # the top interface keeps its pressure and Exner function
        c["exner"][:, -1] = a["exner"][:, -1]
        return dict(dp=c["dp"], pres=c["pres"], exner=c["exner"], tdp=a["tdp"], tlo=a["tlo"], flux=a["flux"],
                    omega=c["omega"])
    if kind == "trcadv":
        for q in range(cfg.ntra):
            tt, tl = a["tt"][q], a["tl"][q]
            x, xdp, tx, lo = _tracer(t, a["tr"][q], a["trdp"][q], a["te"][q], a["flux"][0], a["dp"],
                                     (tt[2], tt[1], tl[2], tl[1]), ab)
            a["tr"][q], a["trdp"][q], tt[0], tl[0] = x, xdp, tx, lo
        return dict(tr=a["tr"], trdp=a["trdp"], tt=a["tt"], tl=a["tl"])
    if kind == "momtum":
        w = dict(u=a["ue"], v=a["ve"], th=a["the"], mont=a["monte"], uvsq=a["uvsqe"])
        u, v, rv, ut, vt = _momentum(t, cfg, a, w, (a["ut"][2], a["ut"][1], a["vt"][2], a["vt"][1]), ab)
        a["ut"][0], a["vt"][0] = ut, vt
        return dict(u=u, v=v, relvor=rv, ut=a["ut"], vt=a["vt"])
    c = _hybrid(t, cfg, ITS, a)
    tr = torch.stack(c["tr"])
    tr[1:3] = tr[1:3].clamp(min=1e-10)
    n = t.n
    mont, ph = _hydrostatic(c["exner"], tr[0], torch.zeros(n, dtype=F64, device="cuda"))
    psrf = c["dp"].sum(1)
    ptdcy = torch.zeros(2, n, dtype=F64, device="cuda")
    ptdcy[ITS % 2] = psrf - a["psrf"]
    mass = t.area[:, None] * c["dp"]
    return dict(u=c["u"], v=c["v"], tr=tr, sdot=c["sdot"], exner=c["exner"], dp=c["dp"], pres=c["pres"], ph=ph,
                mont=mont, trdp=tr * c["dp"], psrf=psrf, ptdcy=ptdcy,
                qtrcr=np.array([float((mass * x).sum()) for x in tr]), qmass=float(mass.sum()) / GRAV)


def work(case):
    """Every input read once and every output written once (grid tables too)."""
    n, L, T, m = 10 * 4 ** case["glvl"] + 2, case["nvl"], case["ntra"], case["members"]
    esz = 8 if case["prec"] == "f64" else 4
    words, table, flops = {
        # the state, both old AB3 slots in, the new one and the state out
        "step": (29 + 10 * T, 170, 1200 + 260 * T),
        "edges": (41 + 7 * T, 100, 500 + 80 * T),
        "cnuity": (43, 56, 260),
        "trcadv": (7 + 16 * T, 20, 180 * T),
        "momtum": (43, 80, 340),
        "column": (12 + 3 * T, 14, 300 + 25 * T),
    }[case["kind"]]
    return {"bytes": float(esz) * n * (L * words * m + table), "flops": float(flops) * n * L * m}
