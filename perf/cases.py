"""The work a user of this package has it do, as measurable cases.

A case is one pass through the public interface: the state of a domain is handed over from
device arrays (``Mimica.upload_device``, the hand-over of a GPU-resident host model), the
integrator runs some steps (``Mimica.stepping``, ``Ensemble.step``), and the state comes back
whole (``Mimica.download_device``).  The adjoint case keeps its state resident and moves the
cost's derivative and the gradient through ``Mimica.traj_adjoint``, whose interface is host
arrays.  Inputs are seeded synthetic fields with the distributions of the package's own
benchmark configurations (``fdd3260_b200.config``): the dry warm bubble and the
shallow-cumulus-like layer.

``exact`` restates one integrator step in plain torch FP64 (interior arrays, periodic shifts)
for the WENO and MUSCL schemes, and its reverse-mode derivative through torch autograd for the
adjoint case.
"""
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from fdd3260_b200 import Mimica, config
from fdd3260_b200 import ensemble as ens

F64 = torch.float64
DEV = "cuda"


# ---- the cases ----
def _case(name, flow, maxx, maxy, nz, steps, form="fp64", scheme="weno", extra=0, tracers="smooth", sgs=False,
          graph=True, checks=False, call="step"):
    c = {"flow": flow, "maxx": maxx, "maxy": maxy, "nz": nz, "steps": steps, "form": form, "scheme": scheme,
         "extra": extra, "tracers": tracers, "sgs": sgs, "graph": graph, "checks": checks, "call": call}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a time loop at the smallest useful size: one step, then the per-step checks, as the
        # reference's modelctl loop calls them; eager launches, a host read-back per step
        _case("loop_40x24x30", "bubble", 40, 24, 30, 10, extra=1, graph=False, checks=True),
        # the plain FP64 warm bubble of 64^3 with one passive scalar, ten steps
        _case("bubble_64", "bubble", 64, 64, 64, 10, extra=1),
        # a medium dry domain, the size the adjoint workload runs forward
        _case("bubble_128x96", "bubble", 128, 128, 96, 4, extra=0),
        # ragged sizes (tiles cut at both edges, radices 2, 3 and 5), MUSCL, the reference
        # module's default scheme, moist and stretched
        _case("muscl_150x90x71", "cumulus", 150, 90, 71, 4, scheme="muscl", extra=1),
        # PPM on a moist domain of moderate size
        _case("ppm_160x128x64", "cumulus", 160, 128, 64, 2, scheme="ppm", extra=1),
        # an LES of moderate size with Smagorinsky-Lilly diffusion and surface fluxes
        _case("sgs_192x192x96", "cumulus", 192, 192, 96, 2, extra=0, sgs=True),
        # the mixed form at a moderate size, five scalars
        _case("mixed_256x64", "cumulus", 256, 256, 64, 4, form="mixed", extra=3),
        # many tracers (the capacity configuration's field set: 12 scalars, lognormal tracers)
        _case("tracers12_240x192x96", "cumulus", 240, 192, 96, 2, form="mixed", extra=10, tracers="lognormal"),
        # the headline workload in both arithmetic forms
        _case("cumulus_512_fp64", "cumulus", 512, 512, 256, 2, extra=3),
        _case("cumulus_512_mixed", "cumulus", 512, 512, 256, 2, form="mixed", extra=3),
        # batched members of uneven sizes (the ensemble configuration's size sets)
        {"name": "ensemble_9", "call": "ensemble", "members": 9, "sizes": 3000, "steps": 4, "form": "mixed"},
        # reverse mode: the checkpointed gradient of a final-time cost
        _case("adjoint_128x96", "bubble", 128, 128, 96, 10, extra=0, call="adjoint"),
    ]


_EVEN = sorted(n for n in {2 ** a * 3 ** b * 5 ** c for a in range(1, 9) for b in range(4) for c in range(3)}
               if 16 <= n <= 512)


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["loop", "fp64", "fp64", "mixed", "mixed", "muscl", "ppm", "sgs", "ensemble", "adjoint"])
    if kind == "ensemble":
        return {"call": "ensemble", "members": rng.randint(3, 9), "sizes": rng.randint(1, 9999),
                "steps": rng.choice([2, 3, 4]), "form": rng.choice(["fp64", "mixed"])}
    near = lambda n, cap: min((e for e in _EVEN if e <= cap), key=lambda e: abs(math.log(e / n)))  # noqa: E731
    cap = {"loop": 96, "fp64": 512, "mixed": 512, "muscl": 320, "ppm": 256, "sgs": 320, "adjoint": 144}[kind]
    x = near(_log(rng, 16, cap), cap)
    y = near(x * _log(rng, 0.4, 2.5), cap)
    z = min(int(_log(rng, 16, 256)), 96 if kind in ("loop", "adjoint") else 256)
    cells = x * y * z
    steps = max(1, min(12, int(3e7 / cells)))
    moist = rng.random() < 0.6
    flow = "cumulus" if moist else "bubble"
    if kind == "loop":
        return _case(None, flow, x, y, z, min(steps, 8), extra=rng.randint(0, 2), graph=False, checks=True)
    if kind == "adjoint":
        return _case(None, "bubble", x, y, z, max(2, min(8, int(1.2e7 / cells))), extra=rng.randint(0, 1), call="adjoint")
    if kind == "sgs":
        return _case(None, "cumulus", x, y, z, min(steps, 6), extra=rng.randint(0, 3), sgs=True,
                     form=rng.choice(["fp64", "mixed"]))
    if kind in ("muscl", "ppm"):
        return _case(None, flow, x, y, z, min(steps, 6), scheme=kind, extra=rng.randint(0, 3),
                     form=rng.choice(["fp64", "mixed"]))
    return _case(None, flow, x, y, z, steps, form=kind, extra=rng.randint(0, 8 if cells < 2e7 else 3),
                 tracers=rng.choice(["smooth", "lognormal"]))


# ---- domains and inputs ----
def _domain(c):
    if c["flow"] == "bubble":
        d = config.warm_bubble_domain(c["maxx"], c["maxy"], c["nz"], dx=50.0, dy=50.0, dz=40.0, dt0=0.5, scheme=c["scheme"])
    else:
        d = config.cumulus_domain(c["maxx"], c["maxy"], c["nz"], dx=25.0, dy=25.0, dt0=1.0, scheme=c["scheme"])
    d.precision = {"fp64": 0, "mixed": 1}[c["form"]]
    if c["sgs"]:
        sh = (d.ny, d.nx)
        d.sgs = config.Sgs(pran=-0.4, zdec=2400.0, momsf=1, zrough=1.0, min_w=0.1, esflux=np.full(sh, 7.0e-3),
                           qvflux=np.full(sh, 5.2e-5), mflux=np.full(sh, -(0.28 ** 2)))
    return d


def _col(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=DEV)[:, None, None]


def _profiles(flow, nz):
    """fdz0, dz, pt0, qv0, cell-centre heights of the configurations' columns."""
    if flow == "bubble":
        dz, thick = 40.0, np.full(nz, 40.0)
        return np.ones(nz), dz, np.full(nz, 300.0), np.zeros(nz), np.cumsum(thick) - 0.5 * thick
    dz = 10.0
    thick = 10.0 + 90.0 * 0.5 * (1.0 + np.tanh(((np.arange(nz) + 0.5) / nz - 0.5) / 0.18))
    zc = np.cumsum(thick) - 0.5 * thick
    qt = np.interp(zc, [0.0, 500.0, 1500.0, zc[-1]], [17e-3, 16e-3, 8e-3, 4e-3])
    return thick / dz, dz, 298.0 + 12.0 * zc / zc[-1], qt, zc


def _density(fdz0, dz, pt0, psurf=101600.0):
    """Hydrostatic base-state density at the cell centres (the model's ten-fold recurrence)."""
    g, pref, cp, cv = 9.81, 1.0e5, 1004.0, 716.0
    rho = lambda p, t: p / ((cp - cv) * t * (p / pref) ** ((cp - cv) / cp))  # noqa: E731
    n = len(pt0)
    dz1 = np.append(1.0 / (0.5 * dz * (fdz0[:-1] + fdz0[1:])), 0.0)
    p, den = np.zeros(n), np.zeros(n)
    p[0] = psurf
    for _ in range(10):
        den[0] = rho(p[0], pt0[0])
        p[0] = psurf - g * 0.5 * (rho(psurf, pt0[0]) + den[0]) * 0.5 * dz * fdz0[0]
    for k in range(1, n):
        p[k] = p[k - 1] - g * den[k - 1] / dz1[k - 1]
        for _ in range(10):
            den[k] = rho(p[k], pt0[k])
            p[k] = p[k - 1] - g * 0.5 * (den[k - 1] + den[k]) / dz1[k - 1]
    return den


def _fields(flow, maxx, maxy, nz, extra, tracers, seed, amp=2.0):
    """[u, v, w, p, dens, theta, (qt), tracers...] on the interior, and qt's index among the
    scalars (-1: dry)."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    sh = (nz, maxy, maxx)
    fdz0, dz, pt0, qv0, zc = _profiles(flow, nz)
    uni = lambda a, b: torch.rand(sh, generator=gen, device=DEV, dtype=F64) * (b - a) + a  # noqa: E731
    nrm = lambda s: torch.randn(sh, generator=gen, device=DEV, dtype=F64) * s  # noqa: E731
    dens = _col(_density(fdz0, dz, pt0)).expand(sh).clone()
    zero = torch.zeros(sh, dtype=F64, device=DEV)
    if flow == "bubble":
        x = (torch.arange(maxx, device=DEV, dtype=F64) + 0.5) * 50.0
        y = (torch.arange(maxy, device=DEV, dtype=F64) + 0.5) * 50.0
        lz = nz * 40.0
        rad = min(500.0, 0.25 * lz)
        r = torch.sqrt((x[None, None, :] - 25.0 * maxx) ** 2 + (y[None, :, None] - 25.0 * maxy) ** 2 + (_col(zc) - 0.3 * lz) ** 2)
        th = 300.0 + torch.where(r < rad, amp * torch.cos(math.pi * r / (2 * rad)) ** 2, zero) + uni(-0.01, 0.01)
        u, v, w = uni(-0.1, 0.1), uni(-0.1, 0.1), uni(-0.1, 0.1)
        w[0] = 0.0
        return [u, v, w, zero, dens, th] + [uni(0.0, 1.0) for _ in range(extra)], -1
    low = _col(zc < 500.0).to(F64)
    th = _col(pt0) + low * nrm(0.1)
    qt = torch.clamp(_col(qv0) + low * nrm(1e-4), min=1e-6)
    out = [nrm(0.5) - 8.0, nrm(0.5), zero.clone(), zero, dens, th, qt]
    for e in range(extra):
        scale = (1e-4, 1e5, 1e8)[e % 3]
        if tracers == "lognormal":
            out.append(scale * torch.exp(nrm(1.0)))
        else:
            out.append(scale * torch.exp(-_col(zc) / 1500.0) * (1.0 + low * nrm(0.01)))
    return out, 1


def _halo(a):
    """Interior -> the halo'd layout (three periodic ghost cells low, two high in x and y)."""
    a = torch.cat([a[..., -3:], a, a[..., :2]], dim=-1)
    return torch.cat([a[:, -3:, :], a, a[:, :2, :]], dim=1).contiguous()


def _ptrs(t):
    q = [a.data_ptr() for a in t]
    return {"u": q[0], "v": q[1], "w": q[2], "p": q[3], "dens": q[4], "scal": q[5:]}


def _spec_list(c):
    return ens.ensemble_specs(c["members"], seed=c["sizes"])


def _member_case(s, c):
    return _case(None, "bubble", s.nxy, s.nxy, s.nz, c["steps"], form=c["form"], extra=1)


class _Run:
    """One domain: its context, the input and the output arrays."""

    def __init__(self, c, seed, amp=2.0):
        f, iqt = _fields(c["flow"], c["maxx"], c["maxy"], c["nz"], c["extra"], c["tracers"], seed, amp)
        self.inp = [_halo(a) for a in f]
        del f
        self.model = Mimica(_domain(c), nscal=len(self.inp) - 5, iqt=iqt)
        self.out = [torch.empty_like(a) for a in self.inp]
        self.pin, self.pout = _ptrs(self.inp), _ptrs(self.out)


def prepare(case, seed):
    c = case
    if c["call"] == "ensemble":
        runs = [_Run(_member_case(s, c), 1000 * seed + s.index, s.amp) for s in _spec_list(c)]
        torch.cuda.synchronize()
        return {"case": c, "runs": runs, "ens": ens.Ensemble([r.model for r in runs])}
    r = _Run(c, seed)
    st = {"case": c, "run": r}
    torch.cuda.synchronize()
    if c["call"] == "adjoint":
        r.model.upload_device(r.pin)
        lam = _cost(c, seed, host=True)
        st["lam"] = config.State(*lam[:5], lam[5:], -1)
    return st


def _cost(c, seed, host=False):
    """dJ/dx(T) of a final-time cost on the winds and potential temperature: seeded normal."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed) + 77)
    sh = (c["nz"], c["maxy"], c["maxx"])
    z = torch.zeros(sh, dtype=F64, device=DEV)
    n = lambda: torch.randn(sh, generator=gen, device=DEV, dtype=F64)  # noqa: E731
    lam = [n(), n(), n(), z, z, n()] + [z] * c["extra"]
    return [_halo(a).cpu().numpy() for a in lam] if host else lam


def run(state):
    c = state["case"]
    if c["call"] == "ensemble":
        for r in state["runs"]:
            r.model.upload_device(r.pin)
        state["ens"].step(c["steps"], ntime0=1)
        for r in state["runs"]:
            r.model.download_device(r.pout)
        return [a for r in state["runs"] for a in r.out]
    r = state["run"]
    m = r.model
    if c["call"] == "adjoint":
        g = m.traj_adjoint(state["lam"], c["steps"], ckpt=max(1, c["steps"] // 2))
        return [g.u, g.v, g.w, g.p, g.dens, *g.scal]
    m.upload_device(r.pin)
    told = []
    if c["checks"]:
        for n in range(c["steps"]):
            m.stepping(1, ntime0=n + 1, graph=c["graph"])
            told.append(m.checkall(apply=False)["maxcfl"])
    else:
        m.stepping(c["steps"], ntime0=1, graph=c["graph"])
    m.download_device(r.pout)
    return r.out + told


# ---- the work a pass cannot do without ----
def _step_work(c):
    cells = c["maxx"] * c["maxy"] * c["nz"]
    ns = 1 + (1 if c["flow"] == "cumulus" else 0) + c["extra"]
    face = {"weno": 45, "muscl": 25, "ppm": 70}[c["scheme"]]
    flops = 2 * (ns + 1) * (3 * face + 12) + 2 * 330 + 2 * (10 * math.log2(c["maxx"] * c["maxy"]) + 40)
    if c["sgs"]:
        flops += 250 + 60 * ns
    return 16.0 * (5 + ns) * cells, float(flops) * cells   # every field of the state in and out, per step


def work(case):
    c = case
    if c["call"] == "ensemble":
        w = [_step_work(_member_case(s, c)) for s in _spec_list(c)]
        return {"bytes": c["steps"] * sum(b for b, _ in w), "flops": c["steps"] * sum(f for _, f in w)}
    b, f = _step_work(c)
    if c["call"] == "adjoint":   # forward sweep and reverse sweep, about twice the forward's arithmetic
        return {"bytes": 2 * c["steps"] * b, "flops": 3 * c["steps"] * f}
    return {"bytes": c["steps"] * b, "flops": c["steps"] * f}


# ---- the integrator step in plain torch FP64 ----
class _Ref:
    def __init__(self, c):
        fdz0, self.dz, pt0, qv0, _ = _profiles(c["flow"], c["nz"])
        self.nz, self.maxx, self.maxy = c["nz"], c["maxx"], c["maxy"]
        self.dx, self.dt = (50.0, 0.5) if c["flow"] == "bubble" else (25.0, 1.0)
        self.scheme, self.moist = c["scheme"], c["flow"] == "cumulus"
        dz, n = self.dz, self.nz
        den = _density(fdz0, dz, pt0)
        dz1 = 1.0 / (0.5 * dz * (fdz0[:-1] + fdz0[1:]))
        dz1 = np.append(dz1, dz1[-1])
        av = den.copy()
        av[1:] = (fdz0[1:] * den[1:] + fdz0[:-1] * den[:-1]) / (fdz0[1:] + fdz0[:-1])
        f = fdz0
        stab = np.zeros(n)
        stab[1:-1] = (den[2:] - den[:-2]) / (den[1:-1] * dz * (0.5 * f[2:] + f[1:-1] + 0.5 * f[:-2]))
        stab[0] = (den[1] - den[0]) / (den[0] * 0.5 * dz * (f[1] + f[0]))
        stab[-1] = (den[-1] - den[-2]) / (den[-1] * 0.5 * dz * (f[-1] + f[-2]))
        self.f, self.dz1h, self.stab = f, dz1, stab
        self.dzwh, self.dz1wh = dz * f, 1.0 / (dz * f)
        self.den, self.av, self.dz1, self.dzw, self.dz1w = (_col(a) for a in (den, av, dz1, self.dzwh, self.dz1wh))
        self.ref = _col(pt0 * (1.0 + 0.60243 * qv0))

    # periodic shift: value at +n along x (dim 2) or y (dim 1)
    @staticmethod
    def s(a, dim, n):
        return torch.roll(a, -n, dim) if n else a

    def weno(self, xm, x0, xp, xq, uu, full):
        g1, g2, eps = 1.0 / 3.0, 2.0 / 3.0, 1e-15
        fm, fc, fp = 1.5 * x0 - 0.5 * xm, 0.5 * x0 + 0.5 * xp, 1.5 * xp - 0.5 * xq
        low = torch.where(fm < fc, fm, fc)
        low = torch.where(low < fp, low, fp)
        den = (low - x0) + eps
        one = x0.abs() >= den.abs()
        phi = torch.where(one, torch.ones_like(x0), (x0 / torch.where(one, torch.ones_like(den), den)).abs())
        pos = uu >= 0
        far, cen = phi * (torch.where(pos, fm, fp) - x0) + x0, phi * (fc - x0) + x0
        eo, em = torch.where(pos, x0 - xm, xq - xp) ** 2, (xp - x0) ** 2
        a, b = g1 / (eps + eo) ** 2, g2 / (eps + em) ** 2
        nl = (torch.maximum(eo, em) / (torch.minimum(eo, em) + eps) > 20.0) & full
        wf = torch.where(nl, a / (a + b), torch.full_like(a, g1))
        wc = torch.where(nl, b / (a + b), torch.full_like(a, g2))
        return (wf * far + wc * cen) * uu

    def muscl(self, xm, x0, xp, xq, uu, d, dm, d0, dp, om, op, z=False):
        # slopes on the spacings of their own faces; om, op: the widths the limiter test weighs by
        tol, eps = 1e-9, 1e-18
        sp, sm, sq = (xp - x0) * d0, (x0 - xm) * dm, (xq - xp) * dp
        on = (om * sm.abs() > tol * x0.abs() + eps) | (op * sq.abs() > tol * x0.abs() + eps)
        pos = uu >= 0
        so = torch.where(pos, sm, sq)
        ok = (so.abs() > tol * x0.abs()) & (sp.abs() < so.abs() / tol)
        r = torch.where(ok, sp / torch.where(ok, so, torch.ones_like(so)), torch.ones_like(so))
        sl = torch.where(on, torch.clamp(r, 0.0, 1.0) * so, sp)
        return torch.where(pos, x0 + 0.5 * sl * d, xp - 0.5 * sl * d) * uu

    def advect(self, x, ua, va, wa):
        """-(Tx + Ty + Tz) of one density-weighted field"""
        out = 0.0
        dx, n = self.dx, self.nz
        for dim, vel in ((2, ua), (1, va)):
            uu = self.s(vel, dim, 1)
            q = (self.s(x, dim, -1), x, self.s(x, dim, 1), self.s(x, dim, 2))
            F = self.weno(*q, uu, True) if self.scheme == "weno" else \
                self.muscl(*q, uu, dx, 1 / dx, 1 / dx, 1 / dx, dx, dx)
            out = out - (F - self.s(F, dim, -1)) / dx
        ww = wa[1:]                                     # face k+1/2 of level k = 0 .. n-2
        x0, xp = x[:-1], x[1:]
        xm = torch.cat([x[:1], x[:-2]])
        xq = torch.cat([x[2:], x[-1:]])
        if self.scheme == "weno":
            lv = torch.arange(1, n, device=x.device)[:, None, None]
            F = self.weno(xm, x0, xp, xq, ww, (lv >= 3) & (lv <= n - 3))
            a, b, c, w = x[0], x[1], x[2], ww[0]
            bot = torch.where(w >= 0, 0.5 * a + 0.5 * b, (2 / 3) * (0.5 * a + 0.5 * b) + (1 / 3) * (1.5 * b - 0.5 * c)) * w
            a, b, c, w = x[-3], x[-2], x[-1], ww[-1]
            top = torch.where(w >= 0, (1 / 3) * (1.5 * b - 0.5 * a) + (2 / 3) * (0.5 * b + 0.5 * c), 0.5 * b + 0.5 * c) * w
            F = torch.cat([bot[None], F[1:-1], top[None]])
        else:
            d, f, dz = self.dz1, _col(self.f), self.dz
            d0 = d[:-1]
            dm, dp = torch.cat([d[:1], d[:-2]]), torch.cat([d[1:-1], d[-1:]])
            om, op = torch.cat([f[:1], f[:-2]]) * dz, f[1:] * dz
            # the end faces take the inner slope on their missing side, which the limiter test skips
            xm = torch.cat([(x0 - (xp - x0))[:1], xm[1:]])
            xq = torch.cat([xq[:-1], (xp + (xp - x0))[-1:]])
            dm, dp = torch.cat([d0[:1], dm[1:]]), torch.cat([dp[:-1], d0[-1:]])
            zero = torch.zeros_like(om[:1])
            om, op = torch.cat([zero, om[1:]]), torch.cat([op[:-1], zero])
            F = self.muscl(xm, x0, xp, xq, ww, 1.0 / self.dz1w[:-1], dm, d0, dp, om, op)
        zero = torch.zeros_like(x[:1])
        return out - (torch.cat([F, zero]) - torch.cat([zero, F])) * self.dz1w

    def d4(self, a, dim):
        s = self.s
        return -s(a, dim, 2) + 4 * s(a, dim, 1) - 6 * a + 4 * s(a, dim, -1) - s(a, dim, -2)

    def along(self, u, ut, dim):
        s, dx = self.s, self.dx
        F = 0.5 * (s(ut, dim, 1) + ut) * 0.5 * (s(u, dim, 1) + u)
        A = 0.5 * (s(ut, dim, 2) + ut) * 0.5 * (s(u, dim, 2) + u)
        t = 4 / 3 * (F - s(F, dim, -1)) / dx - 1 / 3 * (A - s(A, dim, -2)) / (2 * dx)
        return t - ut.abs() / dx * self.d4(u, dim) / 16

    def across(self, u, vt, dim, odim):
        """horizontal transport along dim of a component staggered along odim"""
        s, dx = self.s, self.dx
        v = 9 / 8 * 0.5 * (s(vt, odim, -1) + vt) - 1 / 8 * 0.5 * (s(vt, odim, -2) + s(vt, odim, 1))
        F = s(v, dim, 1) * 0.5 * (s(u, dim, 1) + u)
        t = 9 / 8 * (F - s(F, dim, -1)) / dx - 1 / 8 * (s(F, dim, 1) - s(F, dim, -2)) / (3 * dx)
        a = s(vt, odim, -1) + vt
        return t - 0.25 * (a + s(a, dim, 1)).abs() / dx * self.d4(u, dim) / 16

    def upward(self, u, wt, odim, isv):
        s, n, z, r = self.s, self.nz, self.dzw, self.dz1w
        w = 9 / 8 * 0.5 * (s(wt, odim, -1) + wt) - 1 / 8 * 0.5 * (s(wt, odim, -2) + s(wt, odim, 1))
        F = w[1:] * (z[1:] * u[1:] + z[:-1] * u[:-1]) / (z[1:] + z[:-1])
        zero = torch.zeros_like(u[:1])
        F = torch.cat([F, zero])
        t0 = F[:1] * r[:1]
        t1 = 9 / 8 * (F[1:2] - F[:1]) * r[1 if isv else 0] - 1 / 8 * F[2:3] / (z[0] + z[1] + z[2])
        tc = 9 / 8 * (F[2:n - 1] - F[1:n - 2]) * r[2:n - 1] - 1 / 8 * (F[3:n] - F[:n - 3]) / (z[1:n - 2] + z[2:n - 1] + z[3:n])
        tn = -F[n - 2:n - 1] * r[n - 1:]
        t = torch.cat([t0, t1, tc, tn])
        a = s(wt, odim, -1) + wt
        mu = 0.25 * (a[2:n - 2] + a[3:n - 1]).abs() * r[2:n - 2]
        D = -u[4:] + 4 * u[3:-1] - 6 * u[2:-2] + 4 * u[1:-3] - u[:-4]
        return t - torch.cat([zero, zero, mu * D / 16, zero, zero])

    def w_side(self, w, ht, dim):
        s, n, dx = self.s, self.nz, self.dx
        b = 0.5 * (ht[1:] + ht[:-1])                    # level k from k and k-1
        core = 9 / 8 * b[1:n - 2] - 1 / 8 * 0.5 * (ht[3:n] + ht[:n - 3])
        u = torch.cat([b[:1], core, b[n - 2:]])         # levels 1 .. n-1
        w1 = w[1:]
        F = s(u, dim, 1) * 0.5 * (s(w1, dim, 1) + w1)
        t = 9 / 8 * (F - s(F, dim, -1)) / dx - 1 / 8 * (s(F, dim, 1) - s(F, dim, -2)) / (3 * dx)
        a = ht[1:] + ht[:-1]
        t = t - 0.25 * (a + s(a, dim, 1)).abs() / dx * self.d4(w1, dim) / 16
        return torch.cat([torch.zeros_like(w[:1]), t])

    def w_up(self, w, wt):
        n, z, d = self.nz, self.dzw, self.dz1
        F = 0.5 * (wt[1:] + wt[:-1]) * 0.5 * (w[1:] + w[:-1])
        ws, zs = z[1:] + z[:-1], z
        A = (zs[1:-1] * wt[2:] + zs[:-2] * wt[:-2]) * (zs[1:-1] * w[2:] + zs[:-2] * w[:-2]) / ws[:-1] ** 2
        last = (zs[n - 2] * wt[n - 2]) * (zs[n - 2] * w[n - 2]) / ws[n - 2] ** 2
        A = torch.cat([A, last[None]])
        zero = torch.zeros_like(w[:1])
        t1 = 4 / 3 * (F[1:2] - F[:1]) * d[:1] - 1 / 3 * A[1:2] / ws[:1]
        tc = 4 / 3 * (F[2:] - F[1:-1]) * d[1:n - 2] - 1 / 3 * (A[2:] - A[:-2]) / ws[1:n - 2]
        tn = -F[n - 2:] * d[n - 2:n - 1]
        t = torch.cat([zero, t1, tc, tn])
        D = -w[4:] + 4 * w[3:-1] - 6 * w[2:-2] + 4 * w[1:-3] - w[:-4]
        return t - torch.cat([zero, zero, wt[2:n - 2].abs() * d[1:n - 3] * D / 16, zero, zero])

    def poisson(self, rhs):
        mx, my, n = self.maxx, self.maxy, self.nz
        S = torch.fft.rfft2(rhs)
        pi = 3.14159265
        sx = np.sin(pi * np.arange(mx // 2 + 1) / mx) ** 2
        ky = np.arange(my)
        sy = np.sin(pi * np.where(ky < my // 2, ky, ky - my) / my) ** 2
        wv = torch.as_tensor(-4.0 * (sx[None, :] + sy[:, None]) / self.dx ** 2, device=rhs.device)
        wv[0, 0] = 1.0
        d1, dw, st, f, dz = self.dz1h, self.dz1wh, self.stab, self.f, self.dz
        a, c, e = np.zeros(n), np.zeros(n), np.zeros(n)
        h = dz * (0.5 * f[2:] + f[1:-1] + 0.5 * f[:-2])
        a[1:-1] = d1[:-2] * dw[1:-1] - st[1:-1] / h
        c[1:-1] = d1[1:-1] * dw[1:-1] + st[1:-1] / h
        e[1:-1] = -dw[1:-1] * (d1[1:-1] + d1[:-2])
        c[0] = d1[0] * dw[0] + st[0] * d1[0]
        e[0] = -c[0]
        a[-1] = dw[-1] * d1[-2] - st[-1] * d1[-2]
        e[-1] = -a[-1]
        bet = wv + e[0]
        U, gam = [S[0] / bet], [None]
        for k in range(1, n):
            gam.append(c[k - 1] / bet)
            bet = wv + e[k] - a[k] * gam[k]
            U.append((S[k] - a[k] * U[k - 1]) / bet)
        for k in range(n - 2, -1, -1):
            U[k] = U[k] - gam[k + 1] * U[k + 1]
        X = torch.stack(U)
        keep = torch.ones_like(wv)
        keep[0, 0] = 0.0                                # the horizontal mean is removed from the solution
        return torch.fft.irfft2(X * keep, s=(my, mx))

    def project(self, mu, mv, mw, p):
        s, dx, dt = self.s, self.dx, self.dt
        up = torch.cat([mw[1:], torch.zeros_like(mw[:1])])
        div = (s(mu, 2, 1) - mu) / dx + (s(mv, 1, 1) - mv) / dx + (up - mw) * self.dz1w
        q = self.poisson(div / dt / self.den)
        mu = mu - dt * self.den * (q - s(q, 2, -1)) / dx
        mv = mv - dt * self.den * (q - s(q, 1, -1)) / dx
        mw = torch.cat([torch.zeros_like(mw[:1]), mw[1:] - dt * self.av[1:] * (q[1:] - q[:-1]) * self.dz1[:-1]])
        return mu, mv, mw - mw.mean(dim=(1, 2), keepdim=True), p + self.den * q

    def step(self, ntime, u, v, w, p, dens, *scal):
        s, dx, dt, den, av = self.s, self.dx, self.dt, self.den, self.av
        u0, v0, w0 = u * den, v * den, w * av
        old = [dens] + [q * dens for q in scal]
        mu, mv, mw, psi = u0, v0, w0, old
        tm, ts = None, None
        for a, first in ((1.0, True), (0.5, False)):
            ua, va, wa = mu / den, mv / den, mw / av
            T = [self.advect(x, ua, va, wa) for x in psi]
            pp = p / den
            gu = -den * (pp - s(pp, 2, -1)) / dx
            gv = -den * (pp - s(pp, 1, -1)) / dx
            gw = -av * torch.cat([mw[:1] / (dt * av[:1]), (pp[1:] - pp[:-1]) * self.dz1[:-1]])
            es = psi[1] + 0.5 * dt * T[1]
            qt = psi[2] + 0.5 * dt * T[2] if self.moist else torch.zeros_like(es)
            bb = psi[0] * 9.81 * (es / psi[0] * (1.0 + 0.60243 * qt / psi[0]) / self.ref - 1.0)
            gw = gw + torch.cat([bb[:1], 0.5 * (bb[:-1] + bb[1:])])
            M = [gu - self.along(mu, ua, 2) - self.across(mu, va, 1, 2) - self.upward(mu, wa, 2, False),
                 gv - self.across(mv, ua, 2, 1) - self.along(mv, va, 1) - self.upward(mv, wa, 1, True),
                 gw - self.w_side(mw, ua, 2) - self.w_side(mw, va, 1) - self.w_up(mw, wa)]
            tm = M if first else [x + y for x, y in zip(M, tm)]
            ts = T if first else [x + y for x, y in zip(T, ts)]
            psi = [x + a * dt * t for x, t in zip(old, ts)]
            mu, mv, mw, p = self.project(u0 + a * dt * tm[0], v0 + a * dt * tm[1], w0 + a * dt * tm[2], p)
        return [mu / den, mv / den, mw / av, p, psi[0]] + [x / psi[0] for x in psi[1:]]

    def maxcfl(self, f):
        a = max(float(f[0].abs().max()), float(f[1].abs().max())) * self.dt / self.dx
        return max(a, float((f[2].abs() * self.dz1w).max()) * self.dt)


def _pad0(a):
    return torch.nn.functional.pad(a, (3, 2, 3, 2))


def _exact_steps(c, seed, amp=2.0):
    f, _ = _fields(c["flow"], c["maxx"], c["maxy"], c["nz"], c["extra"], c["tracers"], seed, amp)
    r, told = _Ref(c), []
    for n in range(c["steps"]):
        f = r.step(n + 1, *f)
        if c["checks"]:
            told.append(r.maxcfl(f))
    return [_halo(a) for a in f] + told


def exact(case, seed):
    c = case
    if c["call"] == "ensemble":
        with torch.no_grad():
            return [a for s in _spec_list(c) for a in _exact_steps(_member_case(s, c), 1000 * seed + s.index, s.amp)]
    if c["sgs"] or c["scheme"] == "ppm":
        return None
    if c["call"] == "adjoint":
        f, _ = _fields(c["flow"], c["maxx"], c["maxy"], c["nz"], c["extra"], c["tracers"], seed)
        r = _Ref(c)
        x0 = [a.clone().requires_grad_() for a in f]
        x = x0
        for n in range(c["steps"]):
            x = checkpoint(lambda *q, n=n: tuple(r.step(n + 1, *q)), *x, use_reentrant=False)
        J = sum((a * b).sum() for a, b in zip(_cost(c, seed), x))
        return [_pad0(g) for g in torch.autograd.grad(J, x0)]
    with torch.no_grad():
        return _exact_steps(c, seed)
