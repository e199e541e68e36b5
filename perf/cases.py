"""What a user of this framework has it do, as cases that can be timed and compared.

listed() names the cases, draw() gives more of the same ranges; prepare() makes what a
program holds before the call (handles, requests, device fields), run() makes one pass
through the public entry points, work() says what a pass cannot do without, and exact()
gives the pass's results in 64 bits from plain torch.

Kinds of case
  solve    one load step (ep2d_solve_step) or the whole chain (ep2d_compute_eff_moduli)
           from rest, the record or the moduli, and the fields a program saves
  zone     one load step with the plastic zone tracked, then the post-processing of a
           single-pore RVE: polar stresses, static fields, analytic comparison
  batch    several RVEs together (ep2d_batch_solve)
  average  RVE averages of fields a host framework holds on the device
"""
import ctypes
import math
import random

import numpy as np
import torch

import effplast2d_b200 as ep
from effplast2d_b200 import batch as B

SIDE = 20.0          # Lx = Ly
K0, G0, RHO0, CFL = 1.0, 0.5, 1.0, 0.5
SAVED = ("Ux", "Uy", "P", "tauXX", "tauYY", "tauXY")
VELOCITY = ("Vx", "Vy")
PRECISION = {"fp64": ep.FP64, "mixed": ep.MIXED, "f32": ep.F32_BULK}


def solve(name, nx, ny, nl, pores, niter, check, nts=1, precision="fp64", chain=False, elastic=False):
    return {"name": name, "kind": "solve", "nx": nx, "ny": ny, "nl": nl, "pores": pores, "niter": niter, "check": check,
            "nts": nts, "precision": precision, "chain": chain, "elastic": elastic}


def listed():
    return [
        # averaging for a framework that owns its device memory: the smallest call
        {"name": "average_512", "kind": "average", "nx": 512, "ny": 512, "pores": 3},
        # a first look at a small RVE: three load steps of a few iterations, where launches
        # and host work count
        solve("look_64", 64, 64, 3, 1, 100, 50, chain=True),
        # the elastic 128^2 single-pore RVE solved to 1e-9
        solve("elastic_128", 128, 128, 1, 1, 100_000, 10_000, chain=True, elastic=True),
        # a whole small plastic chain with frequent checkpoints
        solve("chain_128", 128, 128, 3, 2, 10_000, 1000, chain=True),
        # one checkpoint interval of the batched workload's sizes, alone
        solve("plastic_256", 256, 256, 3, 2, 10_000, 10_000),
        solve("mixed_512", 512, 512, 3, 2, 10_000, 10_000, precision="mixed"),
        # a grid that is neither square nor a multiple of anything
        solve("ragged_601x403", 601, 403, 2, 3, 10_000, 10_000),
        # the 1024^2 elastoplastic RVE the headline metric is quoted on: its two preload
        # time steps, one checkpoint interval each
        solve("plastic_1024", 1024, 1024, 2, 3, 10_000, 10_000, nts=2),
        # the 2048^2 RVE with shear, larger than L2: one checkpoint interval
        solve("plastic_2048", 2048, 2048, 3, 4, 10_000, 10_000),
        # the FP32 bulk: an interval in FP32, the last one in FP64
        solve("f32_768", 768, 768, 2, 3, 20_000, 10_000, precision="f32"),
        # homogenisation requests of uneven size solved together in mixed precision
        {"name": "batch_8", "kind": "batch", "count": 8, "smallest": 256, "largest": 768, "niter": 10_000, "check": 10_000},
        # the plastic zone of a single-pore RVE and its post-processing
        {"name": "zone_256", "kind": "zone", "nx": 256, "ny": 256, "nl": 2, "pores": 1, "niter": 2000, "check": 1000},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("solve", "batch", "average", "zone"), (8, 2, 1, 1))[0]
    if kind == "average":
        return {"kind": kind, "nx": _log_uniform(rng, 64, 2048), "ny": _log_uniform(rng, 64, 2048), "pores": rng.randint(1, 4)}
    if kind == "zone":
        n = _log_uniform(rng, 64, 512)
        return {"kind": kind, "nx": n, "ny": n, "nl": rng.randint(2, 3), "pores": 1, "niter": 2000, "check": 1000}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 10), "smallest": rng.choice((128, 256)),
                "largest": rng.choice((512, 768)), "niter": 5000, "check": 5000, "pick": rng.randint(0, 999)}
    nx = _log_uniform(rng, 48, 1700)
    ny = max(48, min(1700, int(nx * math.exp(rng.uniform(-0.5, 0.5)))))
    nl = rng.randint(1, 3)
    check = rng.choice((1000, 2500, 5000))
    return {"kind": kind, "nx": nx, "ny": ny, "nl": nl, "pores": rng.randint(1, 4), "niter": 2 * check, "check": check,
            "nts": 1, "precision": rng.choices(("fp64", "mixed", "f32"), (6, 2, 1))[0], "chain": max(nx, ny) < 256,
            "elastic": nl == 1}


# ---- inputs ---------------------------------------------------------------------------
def _pa(nx, ny, y, porosity, pores):
    """the eleven values of pa.dat (get_sigma_2D.m:3-32)"""
    dx, dy = SIDE / (nx - 1), SIDE / (ny - 1)
    dt = CFL * min(dx, dy) / math.sqrt((K0 + 4 * G0 / 3) / RHO0)
    rad = math.sqrt(porosity * SIDE * SIDE / (math.pi * pores * pores))
    return [dx, dy, dt, K0, G0, RHO0, 4.0 / dt / nx, 4.0 / dt / ny, y * math.sqrt(2.0), rad, float(pores)]


def _inputs(case, seed):
    """material, pore and load parameters, from the distributions of the batched workload"""
    rng = random.Random(seed)
    porosity = rng.uniform(0.005, 0.05)
    if case.get("elastic"):
        return _pa(case["nx"], case["ny"], 1.0, 0.2 * porosity, case["pores"]), -rng.uniform(2e-5, 8e-5), [1.0, 1.0, 0.0]
    y = math.exp(rng.uniform(math.log(5e-6), math.log(5e-5)))
    lt = [1.0, 1.0, 0.0] if case["pores"] == 1 else [1.0, rng.uniform(0.6, 1.0), rng.uniform(0.1, 0.5)]
    return _pa(case["nx"], case["ny"], y, porosity, case["pores"]), -rng.uniform(4e-5, 8e-5), lt


def _fields(case):
    """What a program reads back: what the CLI saves and, where it goes on iterating from
    the state, the velocities.  A whole chain ends there, and an elastic RVE's velocities
    have decayed to rounding noise."""
    return SAVED if case.get("chain") or case.get("elastic") else SAVED + VELOCITY


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        rng = random.Random(1000 * seed + case.get("pick", 0))
        sides = [n for n in (128, 256, 384, 512, 768) if case["smallest"] <= n <= case["largest"]]
        specs = []
        for k in range(case["count"]):
            n = sides[(3 * k + case.get("pick", 0)) % len(sides)]  # the same sizes for every seed
            pores = 1 + k % 4
            pa, load, lt = _inputs({"nx": n, "ny": n, "pores": pores}, rng.randrange(1 << 30))
            specs.append(B.spec(n, pa, 2 + k % 2, 1, load, lt))
        return {"kind": kind, "specs": specs, "niter": case["niter"], "check": case["check"]}
    if kind == "average":
        nx, ny = case["nx"], case["ny"]
        pa = _pa(nx, ny, 1e-5, 0.02, case["pores"])
        g = torch.Generator(device="cuda").manual_seed(seed)
        dims = {"P": (ny, nx), "tauXX": (ny, nx), "tauYY": (ny, nx), "tauXY": (ny - 1, nx - 1), "Ux": (ny, nx + 1), "Uy": (ny + 1, nx)}
        dev = {}
        for f, d in dims.items():  # a mean stress or a strain field, with fluctuations about it
            t = 1e-5 * torch.randn(d, dtype=torch.float64, device="cuda", generator=g)
            if f == "P":
                t += 4e-5
            elif f == "Ux":
                t += -6e-5 * pa[0] * torch.arange(nx + 1, dtype=torch.float64, device="cuda")[None, :]
            elif f == "Uy":
                t += -5e-5 * pa[1] * torch.arange(ny + 1, dtype=torch.float64, device="cuda")[:, None]
            dev[f] = t
        return {"kind": kind, "nx": nx, "ny": ny, "pa": (ctypes.c_double * 11)(*pa), "dev": dev,
                "out": torch.zeros(11, dtype=torch.float64, device="cuda")}
    pa, load, lt = _inputs(case, seed)
    s = ep.Solver(case["nx"], case["ny"], pa, nl=case["nl"], niter=case["niter"], eiter=1e-9, check_every=case["check"],
                  precision=PRECISION[case.get("precision", "fp64")])
    return {"kind": kind, "solver": s, "load": load, "lt": lt, "nts": case.get("nts", 1), "chain": case.get("chain", False),
            "fields": _fields(case)}


# ---- one pass -------------------------------------------------------------------------
def _moduli(m):
    return [m["kphi"], m["kd"], m["g"]]


def run(state):
    kind = state["kind"]
    if kind == "average":
        d, vp = state["dev"], ctypes.c_void_p
        rc = ep.lib().ep2d_average_fields_noalloc(state["nx"], state["ny"], state["pa"],
                                                  *[vp(d[f].data_ptr()) for f in ("P", "tauXX", "tauYY", "tauXY", "Ux", "Uy")],
                                                  vp(state["out"].data_ptr()), vp(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError(ep.lib().ep2d_last_error().decode())
        return state["out"]
    if kind == "batch":
        res, _ = B.batch_solve(state["specs"], niter=state["niter"], check_every=state["check"], precision=ep.MIXED)
        return {"moduli": [_moduli(r["num"]) for r in res], "iterations": np.array([r["total_iterations"] for r in res])}
    s = state["solver"]
    s.reset()
    if kind == "zone":
        s.track_plastic_zone(True)
        rec = s.solve_step(0, state["load"], state["lt"])[0]
        out = s.polar_fields(state["load"])
        out.update(s.static_fields())
        out.update(s.analytic_fields(rec["delta_p"], rec["tau_infty"]))
        return out
    out = {}
    if state["chain"]:
        r = s.compute_eff_moduli(state["load"], state["lt"], state["nts"])
        out["moduli"] = _moduli(r["num"])
        out["iterations"] = r["total_iterations"]
    else:
        recs = s.solve_step(0, state["load"], state["lt"], state["nts"])
        out["sigma"] = np.array(recs[-1]["sigma"][:3])
        out["iterations"] = sum(r["iterations"] for r in recs)
    for f in state["fields"]:
        out[f] = s.get(f)
    return out


# ---- what a pass cannot do without ------------------------------------------------------
def _flops_per_cell(nl):
    # stresses 20, return map 45 (NL > 1), momentum and displacement update 20
    return 85 if nl > 1 else 40


def work(case):
    if case["kind"] == "average":
        cells = case["nx"] * case["ny"]
        return {"bytes": 48 * cells + 88, "flops": 45 * cells}
    if case["kind"] == "batch":
        sides = [n for n in (128, 256, 384, 512, 768) if case["smallest"] <= n <= case["largest"]]
        n = [sides[(3 * k + case.get("pick", 0)) % len(sides)] for k in range(case["count"])]
        its = [(2 + k % 2) * case["niter"] for k in range(case["count"])]
        # each load step's displacements are written once by the preload and read once
        return {"bytes": sum(32 * a * a * (i // case["niter"]) for a, i in zip(n, its)),
                "flops": sum(_flops_per_cell(2) * a * a * i for a, i in zip(n, its))}
    cells = case["nx"] * case["ny"]
    if case["kind"] == "zone":
        return {"bytes": (32 + 32 + 33 + 24 + 48) * cells, "flops": _flops_per_cell(2) * cells * case["niter"]}
    steps = case["nl"] if case["chain"] else 1
    # an elastic solve converges after about three intervals
    its = min(case["niter"], 3 * case["check"]) if case["elastic"] else case["niter"] * (case["nts"] + steps - 1)
    # the state written by the preload of each time step and read by its iterations, the
    # saved fields written and copied out
    return {"bytes": (32 * (case["nts"] + steps - 1) + 2 * 8 * len(_fields(case))) * cells, "flops": _flops_per_cell(case["nl"]) * cells * its}


# ---- the same in 64 bits, plain torch -----------------------------------------------------
class _Sim:
    """EffPlast2D.cu's iteration (:3-177) and preload (:349-381) on torch tensors."""

    def __init__(self, nx, ny, pa, nl):
        self.nx, self.ny, self.pa, self.nl = nx, ny, pa, nl
        dx, dy, self.dt, k0, g0, self.rho, self.damp_x, self.damp_y, self.coh, self.rad, self.n = pa
        self.dx, self.dy = dx, dy
        f8 = {"dtype": torch.float64, "device": "cuda"}
        ax = lambda h, cells, count: -0.5 * h * cells + h * torch.arange(count, **f8)  # noqa: E731
        self.xn, self.yn = ax(dx, nx - 1, nx)[None, :], ax(dy, ny - 1, ny)[:, None]
        self.xu, self.yu = ax(dx, nx, nx + 1)[None, :], ax(dy, ny, ny + 1)[:, None]
        self.node = self.in_pore(self.xn, self.yn)
        self.corner = self.in_pore(self.xn[:, :-1] + 0.5 * dx, self.yn[:-1] + 0.5 * dy)
        solid = torch.where(self.node, 0.01, 1.0).to(torch.float64)
        g = g0 * solid
        zero = (~self.node).to(torch.float64)
        self.k, self.g2 = k0 * solid * zero, 2 * g * zero
        self.gc = 0.25 * (g[:-1, :-1] + g[:-1, 1:] + g[1:, :-1] + g[1:, 1:]) * (~self.corner)
        self.ux, self.vx = torch.zeros(ny, nx + 1, **f8), torch.zeros(ny, nx + 1, **f8)
        self.uy, self.vy = torch.zeros(ny + 1, nx, **f8), torch.zeros(ny + 1, nx, **f8)
        self.p, self.txx, self.tyy = (torch.zeros(ny, nx, **f8) for _ in range(3))
        self.txy = torch.zeros(ny - 1, nx - 1, **f8)
        self.tav = torch.zeros(ny, nx, **f8)
        self.yn_hit, self.yc_hit = torch.zeros_like(self.node), torch.zeros_like(self.corner)
        self.strain = [0.0, 0.0, 0.0]
        self.graph = None

    def in_pore(self, x, y):
        n, hit = self.n, None
        lx, ly = self.dx * (self.nx - 1), self.dy * (self.ny - 1)
        for k in range(int(n)):
            for m in range(int(n)):
                a = x - 0.5 * lx * (1.0 - 1.0 / n) + lx / n * k
                b = y - 0.5 * ly * (1.0 - 1.0 / n) + ly / n * m
                h = torch.sqrt(a * a + b * b) < self.rad
                hit = h if hit is None else hit | h
        return hit

    def step(self):
        ux, uy, dx, dy = self.ux, self.uy, self.dx, self.dy
        exx, eyy = (ux[:, 1:] - ux[:, :-1]) / dx, (uy[1:] - uy[:-1]) / dy
        div = exx + eyy
        self.p.copy_(-self.k * div)
        txx, tyy = self.g2 * (exx - div / 3), self.g2 * (eyy - div / 3)
        txy = self.gc * ((ux[1:, 1:-1] - ux[:-1, 1:-1]) / dy + (uy[1:-1, 1:] - uy[1:-1, :-1]) / dx)
        if self.nl > 1:
            quad = lambda t: 0.25 * (t[:-1, :-1] + t[:-1, 1:] + t[1:, :-1] + t[1:, 1:])  # noqa: E731
            tav = torch.nn.functional.pad(quad(txy)[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
            jn = torch.sqrt(txx * txx + tyy * tyy + 2 * tav * tav)
            cx, cy = quad(txx), quad(tyy)
            jc = torch.sqrt(cx * cx + cy * cy + 2 * txy * txy)
            self.yn_hit |= jn > self.coh
            self.yc_hit |= jc > self.coh
            fn = torch.where(jn > self.coh, self.coh / jn, 1.0)
            txx, tyy, txy = txx * fn, tyy * fn, txy * torch.where(jc > self.coh, self.coh / jc, 1.0)
            self.tav.copy_(tav * fn)
        self.txx.copy_(txx)
        self.tyy.copy_(tyy)
        self.txy.copy_(txy)
        sx, sy = txx - self.p, tyy - self.p
        r = self.dt / self.rho
        self.vx[1:-1, 1:-1].mul_(1 - self.dt * self.damp_x).add_(
            r * ((sx[1:-1, 1:] - sx[1:-1, :-1]) / dx + (txy[1:] - txy[:-1]) / dy))
        self.vy[1:-1, 1:-1].mul_(1 - self.dt * self.damp_y).add_(
            r * ((sy[1:, 1:-1] - sy[:-1, 1:-1]) / dy + (txy[:, 1:] - txy[:, :-1]) / dx))
        ux.add_(self.vx, alpha=self.dt)
        uy.add_(self.vy, alpha=self.dt)

    def iterate(self, n):
        if self.graph is None:
            keep = [t.clone() for t in (self.ux, self.uy, self.vx, self.vy)]
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                self.step()
            torch.cuda.current_stream().wait_stream(side)
            self.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(self.graph):
                for _ in range(10):
                    self.step()
            for t, k in zip((self.ux, self.uy, self.vx, self.vy), keep):
                t.copy_(k)
            self.yn_hit.zero_()
            self.yc_hit.zero_()
        for _ in range(n // 10):
            self.graph.replay()
        for _ in range(n % 10):
            self.step()

    def load_step(self, first, lsv, lt, nts, niter, check):
        total = 0
        for it in range(nts):
            d = [lsv * v / nts for v in lt]
            self.strain = [a + b for a, b in zip(self.strain, d)]
            if first and it == 0:
                self.ux.zero_()
                self.uy.zero_()
            self.ux += self.xu * d[0] + self.yn * d[2]
            self.uy += self.yu * d[1] + self.xn * d[2]
            done = 0
            while done < niter:
                n = min(niter, (done // check + 1) * check) - done
                self.iterate(n)
                done += n
                if done % check == 0:
                    v = [float(t.abs().max()) for t in (self.vx, self.vy)]
                    e = (v[0] / (self.dx * (self.nx - 1)) + v[1] / (self.dy * (self.ny - 1))) * self.dt
                    if e / max(abs(self.strain[0]), self.strain[1], self.strain[2]) < 1e-9:
                        break
            total += done
        return total

    def fields(self):
        return dict(zip(SAVED + VELOCITY, (self.ux, self.uy, self.p, self.txx, self.tyy, self.txy, self.vx, self.vy)))


def _exact_average(case, seed):
    st = prepare(case, seed)
    d, nx, ny, pa = st["dev"], case["nx"], case["ny"], list(st["pa"])
    nu = (1.5 * pa[3] - pa[4]) / (3.0 * pa[3] + pa[4])
    p, xx, yy, xy, ux, uy = (d[f] for f in ("P", "tauXX", "tauYY", "tauXY", "Ux", "Uy"))
    inn = (slice(1, ny - 1), slice(1, nx - 1))
    sums = [(xx - p)[inn].sum(), (yy - p)[inn].sum(), xy[1:, 1:].sum() + (nu * (xx + yy - 2 * p))[inn].sum()]
    a, b = int(nx / pa[10]), int(ny / pa[10])
    j, i = torch.arange(b + 1, ny - b, device="cuda"), torch.arange(a + 1, nx - a, device="cuda")
    j, i = j[(j >= 1) & (j < ny - 1)][:, None], i[(i >= 1) & (i < nx - 1)][None, :]
    q = lambda t, dj=0, di=0: t[j + dj, i + di]  # noqa: E731
    per = [(q(xx) - q(p)).sum(), (q(yy) - q(p)).sum(), 0.25 * (q(xy, -1, -1) + q(xy, -1) + q(xy, 0, -1) + q(xy)).sum(),
           nu * (q(xx) + q(yy) - 2 * q(p)).sum()]
    dxy = [q(ux) - q(ux, -1), q(ux, 0, 1) - q(ux, -1, 1), q(ux, 1) - q(ux), q(ux, 1, 1) - q(ux, 0, 1)]
    dyx = [q(uy) - q(uy, 0, -1), q(uy, 0, 1) - q(uy), q(uy, 1) - q(uy, 1, -1), q(uy, 1, 1) - q(uy, 1)]
    eps = [((q(ux, 0, 1) - q(ux)) / pa[0]).sum(), ((q(uy, 1) - q(uy)) / pa[1]).sum(),
           0.125 * (sum(dxy) / pa[1] + sum(dyx) / pa[0]).sum()]
    inner = (nx - 2 * a) * (ny - 2 * b)
    f = lambda v, n: float(v) / n if n else math.copysign(math.inf, float(v)) if float(v) else math.nan  # noqa: E731
    out = [f(sums[0], nx * ny), f(sums[1], nx * ny), f(sums[2], (nx - 1) * (ny - 1)), 0.0] + [f(v, inner) for v in per + eps]
    return torch.tensor(out, dtype=torch.float64)


def _exact_zone(case, seed):
    pa, load, lt = _inputs(case, seed)
    s = _Sim(case["nx"], case["ny"], pa, case["nl"])
    s.load_step(True, load, lt, 1, case["niter"], case["check"])
    nx, ny, coh = s.nx, s.ny, s.coh
    plast = s.yn_hit.to(torch.int32) + torch.nn.functional.pad(s.yc_hit.to(torch.int32), (1, 1, 1, 1)).unfold(0, 2, 1).unfold(1, 2, 1).sum((2, 3))
    r = torch.sqrt(s.xn * s.xn + s.yn * s.yn)
    sn, cs, on = s.yn / r, s.xn / r, (plast > 0) & (r >= s.rad)
    sxx, syy, sgn = s.txx - s.p, s.tyy - s.p, math.copysign(1.0, load)
    polar = {"Snurr": sxx * cs * cs + 2 * s.tav * sn * cs + syy * sn * sn, "Snuff": sxx * sn * sn - 2 * s.tav * sn * cs + syy * cs * cs,
             "Sanrr": sgn * 2 * coh * torch.log(torch.sqrt(r)) / math.sqrt(2.0),
             "Sanff": sgn * 2 * coh * (torch.log(torch.sqrt(r)) + 1) / math.sqrt(2.0)}
    out = {k: torch.where(on, v, 0.0) for k, v in polar.items()}
    out["Plast"] = plast.to(torch.uint8)
    ux, uy = torch.where(s.in_pore(s.xu, s.yn), 0.0, s.ux), torch.where(s.in_pore(s.xn, s.yu), 0.0, s.uy)
    out["UnuAbs"] = torch.sqrt((0.5 * (ux[:, :-1] + ux[:, 1:])) ** 2 + (0.5 * (uy[:-1] + uy[1:])) ** 2)
    quad = lambda t: 0.25 * (t[:-1, :-1] + t[:-1, 1:] + t[1:, :-1] + t[1:, 1:])  # noqa: E731
    cxx, cyy = quad(sxx), quad(syy)
    out["J1nu"], out["J2nu"] = 0.5 * (cxx + cyy), 0.5 * ((cxx - cyy) ** 2 + 4 * s.txy ** 2)
    # the analytic hydrostatic solution about the one pore; the error maps jump where an
    # error passes 0.5, so they have no value here
    tot = (sxx + syy)[:, 1:-1]
    side = (sxx + syy)[1:-1]
    dp = -0.125 * (float(tot[0].sum() + tot[-1].sum()) / (nx - 2) + float(side[:, 0].sum() + side[:, -1].sum()) / (ny - 2))
    d = (s.txx - s.tyy)
    tau = -0.125 * (float(d[0, 1:-1].sum() + d[-1, 1:-1].sum()) / (nx - 2) + float(d[1:-1, 0].sum() + d[1:-1, -1].sum()) / (ny - 2))
    y = coh / math.sqrt(2.0)
    xi = 1.0 if dp > 0 else -1.0
    c0, kappa = s.rad * math.exp(abs(dp) / 2 / y - 0.5), tau / y * xi
    rin = s.rad - 0.5 * y * s.rad * math.exp((dp - y) / y) / G0
    outer = lambda a, b: (a / (c0 * (1 - kappa))) ** 2 + (b / (c0 * (1 + kappa))) ** 2 > 1  # noqa: E731
    inner = lambda a, b: (a / rin) ** 2 + (b / rin) ** 2 > 1  # noqa: E731
    ua = 0.5 * y * s.rad ** 2 * math.exp((dp - y) / y) / (G0 * r)
    out["UanAbs"] = torch.where(outer(s.xn, s.yn) | inner(s.xn, s.yn), ua, 0.0)
    xc, yc = s.xn[:, :-1] + 0.5 * s.dx, s.yn[:-1] + 0.5 * s.dy
    rc = torch.sqrt(xc * xc + yc * yc)
    far = (s.rad / rc) ** 2 * y * math.exp(dp / y - 1)
    near = -2 * xi * y * torch.log(rc / s.rad)
    o, i = outer(xc, yc), inner(xc, yc)
    out["J1an"] = torch.where(o, -dp, torch.where(i, near - xi * y, 0.0))
    out["J2an"] = torch.where(o, 2 * far * far, torch.where(i, 2 * y * y, 0.0))
    return {**{k: v.cpu() for k, v in out.items()}, "errorUabs": None, "errorJ1": None, "errorJ2": None, "stats": None}


def exact(case, seed):
    """None for the batch and for solves that would take plain torch too long."""
    kind = case["kind"]
    if kind == "average":
        return _exact_average(case, seed)
    if kind == "zone":
        return _exact_zone(case, seed)
    cells = case["nx"] * case["ny"] if kind == "solve" else 0
    steps = case.get("nts", 1) + (case["nl"] - 1 if case.get("chain") else 0) if kind == "solve" else 0
    if kind == "batch" or case["precision"] == "f32" or case["niter"] * steps * (150e-6 + 500e-12 * cells) > 16:
        return None  # the FP32 bulk leaves FP32 where its own residual stalls
    pa, load, lt = _inputs(case, seed)
    s = _Sim(case["nx"], case["ny"], pa, case["nl"])
    its = s.load_step(True, load, lt, case["nts"], case["niter"], case["check"])
    out = {}
    if case["chain"]:
        mean = 0.5 * (lt[0] + lt[1])
        for step in range(1, case["nl"]):
            its += s.load_step(False, 0.005 * load, [mean, mean, 0.0] if step == 1 else [lt[0] - mean, lt[1] - mean, lt[2]],
                               1, case["niter"], case["check"])
        out["moduli"] = [None, None, None]  # quotients of small differences of averages: from the fields
    else:
        nu = (1.5 * K0 - G0) / (3 * K0 + G0)
        inn = (slice(1, case["ny"] - 1), slice(1, case["nx"] - 1))
        n, m = case["nx"] * case["ny"], (case["nx"] - 1) * (case["ny"] - 1)
        xx, yy, zz = s.txx - s.p, s.tyy - s.p, nu * (s.txx + s.tyy - 2 * s.p)
        out["sigma"] = np.array([float(xx[inn].sum()) / n, float(yy[inn].sum()) / n, float(s.txy[1:, 1:].sum() + zz[inn].sum()) / m])
    out["iterations"] = its
    out.update({k: v.cpu() for k, v in s.fields().items() if k in _fields(case)})
    return out
