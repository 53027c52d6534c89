"""The calls this framework is timed on, and what each of them has to return.

A pass is what a simulation does between two of its outputs: the hydro state of
every level goes from (page-locked) host memory to the resident tree, a stretch of
coarse steps runs on the device schedule, and the state comes back.  The tree is
uploaded (planned, autotuned) once and kept, as such a program keeps it; only the
fields change from pass to pass.  Three kinds of pass differ: the time step of a
level state that is already on the device (emma_hydro_level_dt_noalloc), the
-DWRADHYD layout, whose tracer enters and leaves through the host tree, and the
drop-in entries on a host tree (clean_new_hydro + HydroSolver), which is host data
by nature.

Box sizes, tree shapes, Courant number and value distributions are those of
emma_b200/configs.py (Sod tube 64^3, turbulent box 128^3, random box 256^3, Sedov
tree 64^3..256^3, cosmology-like tree 128^3..1024^3); a seed gives other fields of
the same distribution on the same tree.

exact(): the same scheme (MUSCL-Hancock, minmod, HLLC with the hybrid pressure
estimate, subcycled levels) in 64 bits on dense grids in torch.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from emma_b200 import OctTree, PREC_FP64, PREC_MIXED, ResidentHydro, clean_new_hydro, configs, HydroSolver, lib
from emma_b200.hydro import options

GAMMA = 5.0 / 3.0
PMIN = 1e-10
CFL = 0.8
FLOPS = 700  # per cell update: one reconstruction, three Riemann solves, the update


def listed():
    return [
        # the level time step of another solver's device-resident state (a 32^3 level): the
        # smallest call there is, launches and one read-back
        {"name": "level dt 32^3", "kind": "dt", "cells": 32768},
        # a small periodic box at the default precision: latency of the step's launches
        {"name": "box 32^3 fp64", "kind": "box", "field": "random", "level": 5, "prec": "fp64", "variant": "plain",
         "steps": 50},
        # the Sod tube, transmissive x, mixed precision
        {"name": "sod 64^3 mixed", "kind": "box", "field": "sod", "level": 6, "prec": "mixed", "variant": "plain",
         "steps": 50},
        # the turbulent box at both precisions
        {"name": "turb 128^3 fp64", "kind": "box", "field": "turb", "level": 7, "prec": "fp64", "variant": "plain",
         "steps": 50},
        {"name": "turb 128^3 mixed", "kind": "box", "field": "turb", "level": 7, "prec": "mixed", "variant": "plain",
         "steps": 50},
        # ... with the reference's production default, the tracked internal energy
        {"name": "turb 128^3 mixed dual", "kind": "box", "field": "turb", "level": 7, "prec": "mixed",
         "variant": "dual", "steps": 50},
        # ... and coupled to gravity
        {"name": "turb 128^3 fp64 gravity", "kind": "box", "field": "turb", "level": 7, "prec": "fp64",
         "variant": "gravity", "steps": 20},
        # the large uniform box of the benchmark's default workload
        {"name": "box 256^3 mixed", "kind": "box", "field": "random", "level": 8, "prec": "mixed",
         "variant": "plain", "steps": 50},
        # a point explosion on a static three-level tree, subcycled
        {"name": "sedov 64-256 fp64", "kind": "sedov", "base": 6, "r1": 0.25, "r2": 0.125, "prec": "fp64",
         "variant": "plain", "steps": 20},
        # the cosmology-like tree: 9.3 M cells on four levels, subcycled, fine levels sparse and ragged
        {"name": "cosmo 128-1024 mixed", "kind": "cosmo", "base": 7, "lmax": 10, "prec": "mixed", "variant": "plain",
         "steps": 10},
        # the ionisation tracer of the -DWRADHYD layout (its state enters and leaves through the
        # host tree, which takes as long as a hundred steps: a longer stretch between outputs)
        {"name": "turb 64^3 fp64 tracer", "kind": "box", "field": "turb", "level": 6, "prec": "fp64",
         "variant": "tracer", "steps": 150},
        # EMMA's own calls on its host tree
        {"name": "drop-in 64^3 fp64", "kind": "dropin", "level": 6, "prec": "fp64", "steps": 8},
    ]


def draw(rng):
    kind = rng.choice(["dt", "box", "box", "box", "sedov", "sedov", "dropin"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "dt":
        return {"kind": "dt", "cells": int(round(2 ** rng.uniform(10, 24.99)))}
    if kind == "box":
        level = rng.choice([3, 4, 5, 6, 7, 7, 8])
        variant = rng.choice(["plain", "plain", "dual", "gravity", "tracer"])
        field = rng.choice(["random", "turb", "sod"] if variant == "plain" else ["random", "turb"])
        if variant == "tracer":
            level = min(level, 6)
        if variant != "plain":
            level = min(level, 7)
        low, most = (5, 8) if (level == 8 and prec == "fp64") else ((60, 180) if variant == "tracer" else (5, 50))
        return {"kind": "box", "field": field, "level": level, "prec": prec, "variant": variant,
                "steps": rng.randint(low, most)}
    if kind == "sedov":
        base = rng.choice([4, 5, 6])
        r1 = round(rng.uniform(0.2, 0.4), 4)
        return {"kind": "sedov", "base": base, "r1": r1, "r2": round(r1 * rng.uniform(0.35, 0.6), 4), "prec": prec,
                "variant": rng.choice(["plain", "plain", "dual", "gravity"]), "steps": rng.randint(3, 20)}
    return {"kind": "dropin", "level": rng.choice([4, 5, 6]), "prec": prec, "steps": rng.randint(4, 16)}


# ------------------------------------------------------------------ trees and sessions
class Session:
    """A tree and its place on the GPU: what a program keeps between passes."""

    def __init__(self, case):
        self.case = case
        kind = case["kind"]
        self.tracer = case.get("variant") == "tracer"
        self.lib = lib("rh" if self.tracer else False)
        trans, self.nsub = 0, 2
        if kind in ("box", "dropin"):
            lev = case["level"]
            self.tree = OctTree(lev, lev, rh=self.tracer)
            if case.get("field") == "sod":
                trans = configs.sod().trans
        else:
            cfg = (configs.sedov(base=case["base"], radii=(case["r1"], case["r2"])) if kind == "sedov"
                   else configs.cosmo(base=case["base"], lmax=case["lmax"]))
            self.tree = cfg.build()
        self.trans = trans
        self.levels = [l for l in range(self.tree.lcoarse, self.tree.lmax + 1) if self.tree.noct(l) > 0]
        self.prec = PREC_MIXED if case["prec"] == "mixed" else PREC_FP64
        self.cells = {}   # per level: flat index (x, y, z) of every cell in list order, on the GPU
        self.start = {}   # cosmology tree: the configuration's own fields, on the GPU
        for l in self.levels:
            n = 1 << l
            ijk = torch.from_numpy(np.floor(self.tree.cell_centres(l) * n).astype(np.int32)).cuda().long()
            self.cells[l] = (ijk[:, 0] * n + ijk[:, 1]) * n + ijk[:, 2]
            if kind == "cosmo":
                self.start[l] = torch.from_numpy(self.tree.get_fields(l)[:5]).cuda()
        self.updates = sum(int((~self.tree.split_mask(l)).sum()) * self.nsub ** (l - self.levels[0])
                           for l in self.levels)
        self.hydro = None

    def upload(self):
        variant = self.case["variant"]
        if self.start:  # the autotuner runs on plausible fields, whatever the tree held last
            for l in self.levels:
                self.tree.set_fields(l, *self.start[l].cpu().numpy())
        self.hydro = ResidentHydro(self.tree, precision=self.prec, trans=self.trans, cfl=CFL,
                                   gravity=variant == "gravity", dual=variant == "dual")


_sessions = {}
_resident = None


def _structure(case):
    return tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "steps")))


def _session(case):
    key = _structure(case)
    if key not in _sessions:
        _sessions[key] = Session(case)
    return _sessions[key]


def _activate(s):
    """One tree is resident at a time: upload this session's unless it is there."""
    global _resident
    if _resident is s:
        return
    if _resident is not None and _resident.hydro is not None:
        _resident.lib.emma_hydro_tree_release(_resident.tree.firstoct)
        _resident.hydro = None
    _resident = s
    if s.case["kind"] == "dropin":
        o = options(s.prec, cfl=CFL)
        if s.lib.emma_hydro_set_options(ctypes.byref(o)) != 0:
            raise RuntimeError("set_options")
    else:
        s.upload()


# ------------------------------------------------------------------ fields
def _gauss(n, gen, slope, kmax):
    """Unit-variance periodic Gaussian field, P(k) ~ k^slope with the filter of configs.turb."""
    k1 = torch.fft.fftfreq(n, d=1.0 / n, device="cuda", dtype=torch.float64)
    k = torch.sqrt(k1[:, None, None] ** 2 + k1[None, :, None] ** 2 + k1[None, None, : n // 2 + 1] ** 2)
    amp = torch.where((k >= 1) & (k <= kmax), torch.clamp(k, min=1.0) ** (slope / 2) *
                      torch.exp(-k * k / (4.0 * kmax * kmax)), torch.zeros_like(k))
    noise = torch.randn((n, n, n), generator=gen, device="cuda", dtype=torch.float64)
    f = torch.fft.irfftn(torch.fft.rfftn(noise) * amp, s=(n, n, n))
    f = f - f.mean()
    return f / f.std()


def _grid_fields(field, n, gen):
    """(5, n^3) d,u,v,w,p of a box."""
    if field == "turb":
        kmax = min(32, n // 2)
        d = torch.exp(_gauss(n, gen, -4.0, kmax))
        v = torch.stack([_gauss(n, gen, -4.0, kmax) for _ in range(3)])
        v = v * (2.0 * math.sqrt(GAMMA / float(d.mean())) / math.sqrt(float((v * v).sum(0).mean())))
        w = torch.cat([d[None], v, torch.ones_like(d)[None]])
    elif field == "sod":
        dr, pr = torch.empty(2, device="cuda", dtype=torch.float64).uniform_(0.1, 0.2, generator=gen).tolist()
        w = torch.zeros((5, n, n, n), device="cuda", dtype=torch.float64)
        w[0], w[4] = dr, pr
        w[0, : n // 2], w[4, : n // 2] = 1.0, 1.0
    else:
        w = torch.rand((5, n, n, n), generator=gen, device="cuda", dtype=torch.float64)
        w[0] += 0.5
        w[1:4] -= 0.5
        w[4] += 0.5
    return w.reshape(5, -1)


def _make_fields(s, seed):
    """Per level (5, cells) in list order; tracer: dX of the level; gravity: its acceleration."""
    case = s.case
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    out, extra = {}, {}
    if case["kind"] in ("box", "dropin"):
        lev = case["level"]
        out[lev] = _grid_fields(case.get("field", "turb"), 1 << lev, gen)[:, s.cells[lev]]
    elif case["kind"] == "sedov":
        e0, d0 = (0.5 + torch.rand(2, generator=gen, device="cuda", dtype=torch.float64)).tolist()
        for l in s.levels:
            n = 1 << l
            w = torch.zeros((5, s.cells[l].numel()), device="cuda", dtype=torch.float64)
            w[0], w[4] = d0, 1e-5
            if l == s.levels[-1]:  # the 8 finest cells touching the centre
                c = s.cells[l]
                hot = torch.ones_like(c, dtype=torch.bool)
                for q in (c // (n * n), (c // n) % n, c % n):
                    hot &= (q == n // 2) | (q == n // 2 - 1)
                w[4, hot] = (GAMMA - 1.0) * (e0 / 8.0) * n ** 3
            out[l] = w
    else:  # the configuration's own fields, perturbed smoothly by a tenth
        n = 1 << s.levels[0]
        g = [0.1 * _gauss(n, gen, -4.0, n // 4).reshape(-1) for _ in range(5)]
        for l in s.levels:
            c, m, sh = s.cells[l], 1 << l, l - s.levels[0]
            b = (((c // (m * m)) >> sh) * n + (((c // m) % m) >> sh)) * n + ((c % m) >> sh)
            w = s.start[l].clone()
            cs = torch.sqrt(GAMMA * w[4] / w[0])
            w[0] *= torch.exp(g[0][b])
            w[4] *= torch.exp(g[4][b])
            for k in (1, 2, 3):
                w[k] += cs * g[k][b]
            out[l] = w
    if case.get("variant") == "tracer":
        x = torch.rand(8, generator=gen, device="cuda", dtype=torch.float64)
        for l in s.levels:
            c, n = s.cells[l].double(), float(1 << l)
            extra[l] = out[l][0] * (0.5 + 0.4 * torch.sin(2 * math.pi * (torch.floor(c / (n * n)) / n + x[0])))
    if case.get("variant") == "gravity":
        ph = (2 * math.pi * torch.rand(3, generator=gen, device="cuda", dtype=torch.float64)).tolist()
        for l in s.levels:
            n = 1 << l
            x, y, z = ((q.double() + 0.5) * (2 * math.pi / n) for q in (s.cells[l] // (n * n), (s.cells[l] // n) % n,
                                                                        s.cells[l] % n))
            extra[l] = 0.5 * torch.stack([torch.sin(y + ph[0]), torch.cos(z + ph[1]), torch.sin(x + y + ph[2])])
    return out, extra


# ------------------------------------------------------------------ passes
def _host(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def _dt_state(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    w = torch.rand((5, case["cells"]), generator=gen, device="cuda", dtype=torch.float64)
    w[0] += 0.5
    w[1:4] -= 0.5
    w[4] += 0.5
    return w


def prepare(case, seed):
    if case["kind"] == "dt":
        return {"case": case, "w": _dt_state(case, seed), "lib": lib(),
                "stream": ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), "dt": ctypes.c_double()}
    s = _session(case)
    _activate(s)
    fields, extra = _make_fields(s, seed)
    st = {"case": case, "session": s}
    if case["kind"] == "dropin":
        lev = case["level"]
        w = fields[lev]
        smax = (torch.sqrt((w[1:4] ** 2).sum(0)) + torch.sqrt(GAMMA * w[4] / w[0])).max()
        st["in"] = {lev: w.cpu().numpy()}
        st["dt"] = 0.3 * 0.5 ** lev / (3.0 * float(smax))
    elif s.tracer:
        st["in"] = {l: fields[l].cpu().numpy() for l in s.levels}
        st["extra"] = {l: extra[l].cpu().numpy() for l in s.levels}
    else:
        st["in"] = {l: _host(fields[l]) for l in s.levels}
        st["extra"] = {l: _host(extra[l]) for l in extra}
        st["out"] = {l: torch.empty(fields[l].shape, dtype=torch.float64, pin_memory=True) for l in s.levels}
    torch.cuda.synchronize()
    return st


def _steps(r, nsub, steps):
    r.tsim = 0.0
    r.adt[:] = 0.0
    r.coarse_step(nsub=nsub)
    for _ in range(steps - 1):
        r.step_async(nsub=nsub)
    return r.time()


def run(state):
    case = state["case"]
    if case["kind"] == "dt":
        rc = state["lib"].emma_hydro_level_dt_noalloc(ctypes.c_void_p(state["w"].data_ptr()), case["cells"], 5, CFL,
                                                      state["stream"], ctypes.byref(state["dt"]))
        if rc != 0:
            raise RuntimeError("level_dt_noalloc: %d" % rc)
        return state["dt"].value
    s = state["session"]
    _activate(s)
    if case["kind"] == "dropin":
        lev, t = case["level"], s.tree
        t.set_fields(lev, *state["in"][lev])
        for _ in range(case["steps"]):
            clean_new_hydro(lev, t.firstoct)
            HydroSolver(lev, t.firstoct, state["dt"])
        return {"field": t.get_fields(lev)}
    r = s.hydro
    if s.tracer:
        for l in s.levels:
            s.tree.set_fields(l, *state["in"][l])
            s.tree.set_tracer(l, state["extra"][l])
        s.lib.emma_hydro_fields_upload(s.tree.firstoct)
        t = _steps(r, s.nsub, case["steps"])
        r.download()
        return {"time": t, "field": {str(l): s.tree.get_fields(l)[:5] for l in s.levels},
                "tracer": {str(l): s.tree.get_tracer(l) for l in s.levels}}
    for l in s.levels:
        r.set_state(l, state["in"][l].numpy())
        if l in state["extra"]:
            s.lib.emma_hydro_set_level_force(l, ctypes.c_void_p(state["extra"][l].data_ptr()))
    t = _steps(r, s.nsub, case["steps"])
    for l in s.levels:
        s.lib.emma_hydro_get_level_state(l, ctypes.c_void_p(state["out"][l].data_ptr()))
    return {"time": t, "field": {str(l): state["out"][l] for l in s.levels}}


# ------------------------------------------------------------------ work and tolerance
@functools.lru_cache(maxsize=None)
def _updates(key):
    """Cell updates of one coarse step (every level subcycled nsub = 2 times its parent)."""
    case = dict(key)
    if case["kind"] in ("box", "dropin"):
        return 8 ** case["level"]
    return _session(case).updates


def work(case):
    """A step reads each cell's five doubles and writes them (plus the tracer, plus three
    planes of accelerations read); every step depends on the whole of the one before."""
    if case["kind"] == "dt":
        return {"bytes": 40 * case["cells"], "flops": 10 * case["cells"]}
    per = 80 + (16 if case.get("variant") == "tracer" else 0) + (24 if case.get("variant") == "gravity" else 0)
    n = _updates(_structure(case)) * case["steps"]
    return {"bytes": per * n, "flops": FLOPS * n}


def tolerance(case):
    """About four times what the passes show against exact(), which sums in another order: fp64 up
    to 3.9e-15 (2-norm) and 1.8e-13 (one value), mixed (24-bit face states and fluxes) up to
    6.2e-7 and 4.9e-4, after 50 steps at 256^3."""
    if case["kind"] == "dt":
        return {"rel": 1e-15, "max": 1e-15}  # one maximum, one quotient
    if case["prec"] == "fp64":
        return {"rel": 2e-14, "max": 1e-12}
    return {"rel": 2.5e-6, "max": 2e-3}


# ------------------------------------------------------------------ exact
def _minmod(m, p):
    return torch.where(m * p > 0, torch.where(m.abs() < p.abs(), m, p), torch.zeros_like(m))


def _froot(p, q):
    """f(p) and f'(p) of one side q = (d, p, a) of the exact Riemann solver."""
    d, pk, a = q
    A, B = 2.0 / ((GAMMA + 1) * d), (GAMMA - 1) / (GAMMA + 1) * pk
    rt = torch.sqrt(A / (B + p))
    ra = (p / pk) ** ((GAMMA - 1) / (2 * GAMMA))
    f = torch.where(p > pk, (p - pk) * rt, 2 * a / (GAMMA - 1) * (ra - 1))
    df = torch.where(p > pk, rt * (1 - (p - pk) / (2 * (B + p))), (p / pk) ** (-(GAMMA + 1) / (2 * GAMMA)) / (d * a))
    return f, df


def _star(dl, ul, pl, al, dr, ur, pr, ar):
    """Hybrid PVRS / two-rarefaction / two-shock star pressure and velocity; Newton where it is negative."""
    dbar, abar = 0.5 * (dl + dr), 0.5 * (al + ar)
    ppv = 0.5 * ((pl + pr) + (ul - ur) * dbar * abar)
    pmax, pmin = torch.maximum(pl, pr), torch.minimum(pl, pr)
    z = (GAMMA - 1) / (2 * GAMMA)
    p_tr = ((al + ar - (GAMMA - 1) / 2 * (ur - ul)) / (al / pl ** z + ar / pr ** z)) ** 5
    u_tr = ul - 2 * al / (GAMMA - 1) * ((p_tr / pl) ** z - 1)
    p0 = torch.clamp(ppv, min=0.0)
    gl = torch.sqrt(2 / ((GAMMA + 1) * dl) / (p0 + (GAMMA - 1) / (GAMMA + 1) * pl))
    gr = torch.sqrt(2 / ((GAMMA + 1) * dr) / (p0 + (GAMMA - 1) / (GAMMA + 1) * pr))
    p_ts = (gl * pl + gr * pr - (ur - ul)) / (gl + gr)
    u_ts = 0.5 * ((ul + ur) + (p_ts - pr) * gr - (p_ts - pl) * gl)
    pv = (pmax / pmin < 2) & (pmin < ppv) & (ppv < pmax)
    tr = ~pv & (ppv < pmin)
    p = torch.where(pv, ppv, torch.where(tr, p_tr, p_ts))
    u = torch.where(pv, 0.5 * ((ul + ur) + (pl - pr) / (dbar * abar)), torch.where(tr, u_tr, u_ts))
    bad = p < 0
    if bool(bad.any()):
        L, R = (dl[bad], pl[bad], al[bad]), (dr[bad], pr[bad], ar[bad])
        du = ur[bad] - ul[bad]
        q = torch.clamp(p_ts[bad], min=1e-10)
        q = torch.where(ppv[bad] < pmin[bad], torch.full_like(q, 1e-10), q)
        for _ in range(10):
            (fl, dfl), (fr, dfr) = _froot(q, L), _froot(q, R)
            dp = (fl + fr + du) / (dfl + dfr)
            for _ in range(60):
                dp = torch.where(q - dp < 0, 0.5 * dp, dp)
            q = torch.where(dp.abs() < 1e-10, q, q - dp)
        (fl, _), (fr, _) = _froot(q, L), _froot(q, R)
        p[bad] = q
        u[bad] = 0.5 * (ul[bad] + ur[bad]) + 0.5 * (fr - fl)
    return p, u


def _energy(W):
    return W[4] / (GAMMA - 1) + 0.5 * W[0] * (W[1] ** 2 + W[2] ** 2 + W[3] ** 2)


def _hllc(L, R, ax):
    """HLLC flux normal to ax of the face states L, R (lists d,u,v,w,p): mass, 3 momenta, energy; then
    the star or upwind state's normal velocity and internal energy, and the upwind side and star flag."""
    al, ar = torch.sqrt(GAMMA * L[4] / L[0]), torch.sqrt(GAMMA * R[4] / R[0])
    ul, ur = L[1 + ax], R[1 + ax]
    ps, us = _star(L[0], ul, L[4], al, R[0], ur, R[4], ar)
    one = torch.ones_like(ps)
    g2 = (GAMMA + 1) / (2 * GAMMA)
    SL = ul - al * torch.where(ps <= L[4], one, torch.sqrt(1 + g2 * (ps / L[4] - 1)))
    SR = ur + ar * torch.where(ps <= R[4], one, torch.sqrt(1 + g2 * (ps / R[4] - 1)))
    cross = SL > SR
    SL, SR = (torch.where(cross, torch.minimum(ul - al, ur - ar), SL),
              torch.where(cross, torch.maximum(ul + al, ur + ar), SR))
    left = (SL >= 0) | (~(SR <= 0) & (us >= 0))
    star = ~((SL >= 0) | (SR <= 0))
    W = [torch.where(left, a, b) for a, b in zip(L, R)]
    S = torch.where(left, SL, SR)
    d, un, p, E = W[0], W[1 + ax], W[4], _energy(W)
    F = [d * un] + [d * un * W[1 + k] + (p if k == ax else 0) for k in range(3)] + [un * (E + p)]
    fact = d * (S - un) / (S - us)
    Es = E / d + (us - un) * (us + p / (d * (S - un)))
    U = [d] + [d * W[1 + k] for k in range(3)] + [E]
    Us = [fact] + [fact * (us if k == ax else W[1 + k]) for k in range(3)] + [fact * Es]
    F = [torch.where(star, f + (b - a) * S, f) for f, a, b in zip(F, U, Us)]
    kin = sum(W[1 + k] ** 2 for k in range(3) if k != ax)
    ebar = torch.where(star, fact * (Es - 0.5 * (us * us + kin)), p / (GAMMA - 1))
    return F, torch.where(star, us, un), ebar, left, star, fact, S, d


def _advance(W, dt, dx, ok=None, dual=False, force=None, X=None):
    """One level update of the dense state W: (flux divergence of U, sum_k of the face terms needed by the
    variants); ok: cells whose faces carry flux (leaves, injected coarse leaves)."""
    D = []
    for ax in range(3):
        D.append([_minmod(q - torch.roll(q, 1, ax), torch.roll(q, -1, ax) - q) for q in W])
    div = D[0][1] + D[1][2] + D[2][3]
    adv = [sum(W[1 + ax] * D[ax][k] for ax in range(3)) for k in range(5)]
    h = -0.5 * dt / dx
    P = [adv[0] + W[0] * div, adv[1] + D[0][4] / W[0], adv[2] + D[1][4] / W[0], adv[3] + D[2][4] / W[0],
         adv[4] + GAMMA * W[4] * div]
    C = [q + h * a for q, a in zip(W, P)]
    dU = [torch.zeros_like(W[0]) for _ in range(5)]
    corr = []  # per axis: flux (times dt/dx) through the - face of every cell
    dUe, divu, dX = (torch.zeros_like(W[0]) for _ in range(3))
    for ax in range(3):
        lo = [c - 0.5 * s for c, s in zip(C, D[ax])]
        hi = [c + 0.5 * s for c, s in zip(C, D[ax])]
        for f in (lo, hi):
            f[4] = torch.clamp(f[4], min=PMIN)
            if force is not None:
                for k in range(3):
                    f[1 + k] = f[1 + k] - 0.5 * dt * force[k]
        L = [torch.roll(q, 1, ax) for q in hi]
        F, us, ebar, left, star, fact, S, d = _hllc(L, lo, ax)
        if X is not None:
            x0 = torch.where(left, torch.roll(X / W[0], 1, ax), X / W[0])
            fx = F[0] * x0  # dX is d x0 throughout the fan: its flux is the mass flux times x0
            dX += (fx - torch.roll(fx, -1, ax)) * dt / dx
        if ok is not None:
            both = ok & torch.roll(ok, 1, ax)
            F = [torch.where(both, f, torch.zeros_like(f)) for f in F]
        for v in range(5):
            dU[v] += (F[v] - torch.roll(F[v], -1, ax)) * (dt / dx)
        if ok is not None:
            corr.append([f * (dt / dx) for f in F])
        if dual:
            fe = us * ebar
            dUe += (fe - torch.roll(fe, -1, ax)) * (dt / dx)
            divu += torch.roll(us, -1, ax) - us
    return dU, corr, dUe, divu, dX


def _update(W, dU, dt, dx, dual=False, dUe=None, divu=None, force=None):
    U = [W[0] + dU[0]] + [W[0] * W[1 + k] + dU[1 + k] for k in range(3)] + [_energy(W) + dU[4]]
    ekin = 0.5 * (U[1] ** 2 + U[2] ** 2 + U[3] ** 2) / U[0]
    p = (GAMMA - 1) * (U[4] - ekin)
    if dual:
        e0 = W[4] / (GAMMA - 1)
        pdiv = (GAMMA - 1) * e0 * divu
        e = e0 + dUe - pdiv * (dt / dx)
        e = torch.where(U[4] - ekin > 0.5 * pdiv ** 2, U[4] - ekin, e)
        p = e * (GAMMA - 1)
    out = [U[0], U[1] / U[0], U[2] / U[0], U[3] / U[0], torch.clamp(p, min=PMIN)]
    if force is not None:
        for k in range(3):
            out[1 + k] = out[1 + k] - force[k] * dt
    return out


def _cfl(W, dx, has=None):
    s = torch.sqrt(W[1] ** 2 + W[2] ** 2 + W[3] ** 2) + torch.sqrt(GAMMA * W[4] / W[0])
    if has is not None:
        s = torch.where(has, s, torch.zeros_like(s))
    return CFL * dx / (3 * float(s.max()))


def _exact_box(s, case, fields, extra, steps, dt_fixed=None):
    lev = case["level"]
    n, cells, variant = 1 << lev, s.cells[lev], case.get("variant", "plain")
    dx = 0.5 ** lev

    def grid(plane):
        g = torch.empty(n ** 3, device="cuda", dtype=torch.float64)
        g[cells] = plane
        return g.reshape(n, n, n)

    W = [grid(q) for q in fields[lev]]
    force = [grid(q) for q in extra[lev]] if variant == "gravity" else None
    X = grid(extra[lev]) if variant == "tracer" else None
    pad = 2 if case.get("field") == "sod" else 0  # transmissive x: two copies of the boundary cells
    t = 0.0
    for _ in range(steps):
        dt = dt_fixed if dt_fixed is not None else _cfl(W, dx)
        V = [torch.cat([q[:1].expand(pad, n, n), q, q[-1:].expand(pad, n, n)]) for q in W] if pad else W
        dU, _, dUe, divu, dX = _advance(V, dt, dx, dual=variant == "dual", force=force, X=X)
        if pad:
            dU = [q[pad:-pad] for q in dU]
        W = _update(W, dU, dt, dx, variant == "dual", dUe, divu, force)
        if X is not None:
            X = torch.minimum(torch.clamp(X + dX, min=0.0), W[0])
        t += dt
    back = [q.reshape(-1)[cells] for q in W]
    return t, torch.stack(back), (X.reshape(-1)[cells] if X is not None else None)


class _Dense:
    """A subcycled tree on dense grids: per level the state, which cells exist, which are split."""

    def __init__(self, s, fields):
        self.levels, self.W, self.has, self.split, self.C = s.levels, {}, {}, {}, {}
        self.adt = {l: 0.0 for l in range(s.levels[0] - 1, s.levels[-1] + 1)}
        for l in s.levels:
            n = 1 << l
            w = torch.ones((5, n ** 3), device="cuda", dtype=torch.float64)
            w[:, s.cells[l]] = fields[l]
            has = torch.zeros(n ** 3, device="cuda", dtype=torch.bool)
            has[s.cells[l]] = True
            sp = torch.zeros(n ** 3, device="cuda", dtype=torch.bool)
            sp[s.cells[l]] = torch.from_numpy(s.tree.split_mask(l)).cuda()
            self.W[l] = list(w.reshape(5, n, n, n))
            self.has[l], self.split[l] = has.reshape(n, n, n), sp.reshape(n, n, n)

    @staticmethod
    def up(q):
        for ax in range(3):
            q = q.repeat_interleave(2, ax)
        return q

    @staticmethod
    def down(q):
        n = q.shape[0] // 2
        return q.reshape(n, 2, n, 2, n, 2).sum((1, 3, 5))

    def filled(self, l):
        """The level's state, coarser leaves injected where it has no cells."""
        if l == self.levels[0]:
            return self.W[l]
        return [torch.where(self.has[l], q, self.up(c)) for q, c in zip(self.W[l], self.filled(l - 1))]

    def solve(self, l, dt):
        dx, W = 0.5 ** l, self.filled(l)
        sp, has = self.split[l], self.has[l]
        dU, corr, _, _, _ = _advance(W, dt, dx, ok=~sp)
        if l in self.C:
            dU = [a + b for a, b in zip(dU, self.C[l])]
        new = _update(W, dU, dt, dx)
        leaf = has & ~sp
        if l > self.levels[0]:  # the flux through faces shared with a coarser leaf, for that leaf
            for ax in range(3):
                for v in range(5):
                    f = corr[ax][v]
                    here = leaf & ~torch.roll(has, 1, ax)          # coarse cell across the - face
                    c = torch.roll(torch.where(here, -f, torch.zeros_like(f)), -1, ax)
                    there = torch.roll(leaf, 1, ax) & ~has          # coarse cell on the + side of the face
                    c = c + torch.where(there, f, torch.zeros_like(f))
                    self.C[l - 1][v] += self.down(c) * 0.125
        for v in range(5):
            q = torch.where(leaf, new[v], W[v])
            if l < self.levels[-1]:
                q = torch.where(sp, self.down(self.W[l + 1][v]) * 0.125, q)
            self.W[l][v] = q

    def advance(self, l, tloc):
        adt, lc, dt, count = self.adt, self.levels[0], 0.0, 0
        while True:
            if l < self.levels[-1]:
                self.C[l] = [torch.zeros_like(q) for q in self.W[l]]
            adt[l] = min(1e9, _cfl(self.W[l], 0.5 ** l, self.has[l]))
            if l == lc:
                adt[l - 1] = adt[l]
            adt[l] = adt[l - 1] if adt[l - 1] < adt[l] else min(adt[l], adt[l - 1] - dt)
            if l < self.levels[-1]:
                adt[l] = self.advance(l + 1, tloc)
                if l == lc:
                    adt[l - 1] = adt[l]
            self.solve(l, adt[l])
            dt += adt[l]
            tloc += adt[l]
            count += 1
            if not (dt < adt[l - 1] and count < 2):
                return dt


def exact(case, seed):
    if case["kind"] == "dt":
        w = _dt_state(case, seed).cpu().numpy()
        s = np.sqrt(w[1] ** 2 + w[2] ** 2 + w[3] ** 2) + np.sqrt(GAMMA * w[4] / w[0])
        return CFL * 0.5 ** 5 / (3.0 * float(s.max()))
    s = _session(case)
    if case["kind"] == "dropin":
        dt = prepare(case, seed)["dt"]
    fields, extra = _make_fields(s, seed)
    if case["kind"] == "dropin":
        _, w, _ = _exact_box(s, case, fields, extra, case["steps"], dt)
        a = torch.sqrt(GAMMA * w[4] / w[0])
        return {"field": torch.cat([w, a[None], _energy(w)[None]])}
    if case["kind"] == "box":
        t, w, x = _exact_box(s, case, fields, extra, case["steps"])
        out = {"time": t, "field": {str(case["level"]): w}}
        if x is not None:
            out["tracer"] = {str(case["level"]): x}
        return out
    if case["kind"] == "cosmo" or case["variant"] != "plain":
        return None  # 1024^3 dense grids; the coupled variants' coarse-fine interpolation
    g = _Dense(s, fields)
    t = 0.0
    for _ in range(case["steps"]):
        g.advance(s.levels[0], t)
        t += g.adt[s.levels[0]]
    return {"time": t, "field": {str(l): torch.stack([q.reshape(-1)[s.cells[l]] for q in g.W[l]]) for l in s.levels}}
