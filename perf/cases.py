"""The workloads whose speed is kept track of, as a program that uses the package runs them.

Four kinds of case, each through the package's public entry points:

* ``solve``: one model on one GPU (`Solver`).  ``whole`` cases are one forward solve of
  an inversion loop: the next candidate fault goes up (which puts the model back to its
  initial state), all time steps run, and the history files, the seismograms and the final
  fault planes are read.  The others are the next stretch of a long run: the steps up
  to the next read-back, then the records that they made.
* ``once``: a solve from nothing, as a command-line run does it: context, medium and fault
  up, all steps, final planes read, context closed.
* ``batch``: many models of uneven size in one arena (`Batch`), from their initial
  state to their last step, final planes read.
* ``serve``: a burst of requests of mixed size through the continuous-batching loop.

Grids, friction set-ups, step sizes and sampling are those of the package's named workloads
(`configs.sw_small`, `sw_large`, `fvw_medium`, `batch_model`, `tiny_sw`, `tiny_fvw`), sizes
between them, and the same with odd extents.  The wave field stays on the device, as
in a production run: what a run yields is its fault-plane histories, its seismograms and
its final planes.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fd3d_tsn_b200 import configs
from fd3d_tsn_b200.batch import Batch, bytes_needed
from fd3d_tsn_b200.serve import serve
from fd3d_tsn_b200.solver import Solver

HISTORIES = ("sliprateX", "sliprateZ", "shearstressX", "shearstressZ", "psi")
FINALS = ("slipX", "slipZ", "ruptime", "rise", "sliptime")


def _solve(name, nx, ny, nz, h, steps, stride, law="sw", precision="f32", fspace=False, medium="layers", whole=True,
           kind="solve"):
    return dict(name=name, kind=kind, law=law, nx=nx, ny=ny, nz=nz, h=h, steps=steps, stride=stride,
                precision=precision, fspace=fspace, medium=medium, whole=whole)


def listed():
    return [
        # the smallest model in use (parity and convergence studies): every launch counts
        _solve("sw_tiny", 40, 14, 28, 200.0, 60, 1),
        # one candidate of a slip-weakening inversion, 8 s simulated, records every 0.08 s
        _solve("sw_small", 160, 80, 120, 200.0, 960, 10),
        # the all-double build on an odd grid (checks of the single-precision results)
        _solve("sw_odd_f64", 101, 47, 73, 200.0, 200, 5, precision="f64"),
        # the full-space build (a fifth absorbing strip on top), odd extents
        _solve("sw_fullspace_odd", 197, 61, 93, 200.0, 200, 5, fspace=True),
        # a 3-D velocity model from tomography: nothing can be read per plane
        _solve("sw_medium3d", 400, 200, 200, 100.0, 40, 10, medium="3d", whole=False),
        # one candidate of a rate-and-state study
        _solve("fvw_small", 150, 50, 75, 200.0, 250, 5, law="fvw"),
        # rate-and-state production run, records every 5 steps
        _solve("fvw_medium", 600, 300, 400, 100.0, 20, 5, law="fvw", whole=False),
        # slip-weakening production run: 214 M cells, 5 layers
        _solve("sw_large", 1000, 400, 500, 50.0, 20, 5, whole=False),
        # one command-line run of a model of the batch's size, 8 s simulated
        _solve("sw_once", 140, 30, 80, 200.0, 960, 10, kind="once"),
        # an ensemble of candidates that fills the GPU, 2 s simulated
        dict(name="batch_64", kind="batch", models=64, mix=2024, steps=240, schedule="graph"),
        # a handful of candidates at a time, as a sampler with few chains proposes them
        dict(name="batch_4", kind="batch", models=4, mix=7, steps=240, schedule="persistent"),
        # a burst of requests to the solve service, the largest twice as fine
        dict(name="serve_12", kind="serve", requests=12, mix=4242, steps=240),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve"] * 8 + ["once", "batch", "batch", "serve"])
    if kind == "batch":
        return dict(kind=kind, models=_log(rng, 2, 64), mix=rng.randrange(1 << 20), steps=_log(rng, 40, 240),
                    schedule=rng.choice(["graph", "graph", "persistent"]))
    if kind == "serve":
        return dict(kind=kind, requests=_log(rng, 3, 16), mix=rng.randrange(1 << 20), steps=_log(rng, 60, 240))
    if kind == "once":
        return _unnamed(_solve("", _log(rng, 100, 180), _log(rng, 20, 40), _log(rng, 60, 100), 200.0,
                               _log(rng, 100, 960), 10, kind=kind))
    law = rng.choice(["sw", "sw", "fvw"])
    precision = rng.choice(["f32"] * 5 + ["f64"])
    top = 0.6 if precision == "f64" else 1.0  # the double build takes twice the memory and time
    nx, ny, nz = (_log(rng, lo, lo + top * (hi - lo)) for lo, hi in ((40, 900), (14, 360), (28, 450)))
    cells = (nx + 20) * (ny + 10) * (nz + 12)
    whole = cells < 4e6
    stride = rng.choice([1, 2, 5]) if cells < 1e5 else rng.choice([5, 10])
    steps = max(2, min(400 if whole else 80, int((4e8 if whole else 2e9) / cells) // stride)) * stride
    steps = min(steps, 20 * stride if not whole else 800)
    h = 200.0 if nz < 150 else 100.0 if nz < 300 else 50.0
    return _unnamed(_solve("", nx, ny, nz, 100.0 if law == "fvw" and h == 50.0 else h, steps, stride, law=law,
                           precision=precision, fspace=rng.random() < 0.2,
                           medium="3d" if law == "sw" and rng.random() < 0.3 else "layers", whole=whole))


def _unnamed(case):
    del case["name"]
    return case


# ---------------------------------------------------------------- inputs
def _model(c, seed):
    if c["law"] == "fvw":
        m = configs.fvw_model(c["nx"], c["ny"], c["nz"], c["h"], 1.0, seed, history_stride=c["stride"],
                              precision=c["precision"], ntfd=1 << 20, fspace=c["fspace"],
                              fault_m=(0.8 * c["nx"] * c["h"], 0.7 * c["nz"] * c["h"]))
    else:
        lay = configs.layered(np.random.default_rng(seed + 1000), 5, c["nz"] * c["h"])
        m = configs.sw_model(c["nx"], c["ny"], c["nz"], c["h"], 1.0, seed, layers=lay, history_stride=c["stride"],
                             precision=c["precision"], ntfd=1 << 20, fspace=c["fspace"], corr_m=10 * c["h"],
                             dc_patch_m=20 * c["h"], dc_range=(0.3, 0.6))
    m["history_capacity"] = max(8, c["steps"] // c["stride"])
    return m


def _medium3d(m, seed):
    """The layered medium with smooth 3-D slow anomalies of up to 10% in wave speed, as float32
    arrays in the order a Fortran host holds them."""
    g = torch.Generator().manual_seed(seed + 77)
    n = (m["nzt"], m["nyt"], m["nxt"])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    coarse = torch.rand((1, 1, *(max(2, k // 12) for k in n)), generator=g).to(dev)
    f = 1.0 - 0.1 * torch.nn.functional.interpolate(coarse, size=n, mode="trilinear", align_corners=True)[0, 0]
    lam, mu, d = (torch.as_tensor(a, dtype=torch.float32, device=dev).view(-1, 1, 1) for a in m["medium"])
    return [t.contiguous().cpu().numpy().T for t in (lam * f * f, mu * f * f, d * (0.5 + 0.5 * f))]


def _mixed(c, seed, n):
    """Models of uneven size (configs.batch_model's ranges); the sizes belong to the case, the
    faults to the seed."""
    sizes = np.random.default_rng(c["mix"])
    out = []
    for q in range(n):
        fx, fz = int(round(sizes.uniform(8e3, 24e3) / 200.0)), int(round(sizes.uniform(6e3, 14e3) / 200.0))
        h = 100.0 if c["kind"] == "serve" and q == n - 1 else 200.0
        if h == 100.0:
            fx, fz = 2 * fx, 2 * fz
        out.append(configs.sw_model(fx + 60, 30, fz + 30, h, 1.0, seed * 1000 + q, patch_nodes=(fx, fz), nstations=2,
                                    ntfd=c["steps"]))
        out[-1]["request"] = q
    return out


def prepare(case, seed):
    c = case
    if c["kind"] == "batch":
        models = _mixed(c, seed, c["models"])
        b = Batch(int(sum(bytes_needed(m) for m in models) * 1.05) + (64 << 20), len(models) + 4)
        slots = [b.add(m) for m in models]
        b.set_schedule(c["schedule"])
        b.set_tuning(32 if c["schedule"] == "graph" else 8, 0)
        return dict(case=c, batch=b, slots=slots)
    if c["kind"] == "serve":
        models = _mixed(c, seed, c["requests"])
        return dict(case=c, stream=[(0.0, m) for m in models],
                    budget=int(sum(bytes_needed(m) for m in models) * 0.6) + max(bytes_needed(m) for m in models))
    m = _model(c, seed)
    if c["kind"] == "once":
        return dict(case=c, model=m)
    s = Solver(m)
    if c["medium"] == "3d":
        s.upload_medium_arrays(*_medium3d(m, seed), real_kind=4)
    return dict(case=c, model=m, solver=s)


# ---------------------------------------------------------------- one pass
def _records(s, c, nrec):
    rec0 = s.history_records() - nrec
    kind = 8 if c["precision"] == "f64" else 4
    out = {f: s.history(f, rec0, nrec, real_kind=kind) for f in HISTORIES[:s.nf]}
    out["stations"] = s.stations(rec0, nrec)
    return out


def _joined(finals):
    return {k: np.concatenate([f[k].ravel(order="F") for f in finals]) for k in FINALS}


def run(state):
    c = state["case"]
    if c["kind"] == "batch":
        b = state["batch"]
        for s in state["slots"]:
            b.reset(s)
        b.run(c["steps"])
        b.sync()
        return _joined([b.final(s) for s in state["slots"]])
    if c["kind"] == "serve":
        results, _ = serve(state["stream"], state["budget"], chunk=32,
                           tuning=dict(schedule="graph", kchunk=32, ctas_per_sm=0))
        return _joined([r.final for r in sorted(results, key=lambda r: r.request)])
    if c["kind"] == "once":
        s = Solver(state["model"])
        s.run(c["steps"])
        s.sync()
        out = s.final()
        s.close()
        return out
    s = state["solver"]
    if c["whole"]:
        s.upload_fault(state["model"]["fault"])
    s.run(c["steps"])
    s.sync()
    out = _records(s, c, c["steps"] // c["stride"])
    if c["whole"]:
        out.update(s.final())
    return out


# ---------------------------------------------------------------- what a pass cannot do without
def _grids(c):
    """(nxt, nyt, nzt, interior cells, absorbing-strip cells, fault nodes) of the case's models."""
    if c["kind"] in ("batch", "serve"):
        models = _mixed(c, 0, c.get("models", c.get("requests")))
        sizes = [(m["nxt"] - 20, m["nyt"] - 10, m["nzt"] - 12) for m in models]
    else:
        sizes = [(c["nx"], c["ny"], c["nz"])]
    for nx, ny, nz in sizes:
        full = bool(c.get("fspace"))
        nxt, nyt = nx + 20, ny + 10
        pml = 2 * 9 * ny * nz + (nxt - 2) * 9 * nz + (nxt - 2) * (nyt - 1) * 9 * (2 if full else 1)
        yield nxt, nyt, nz + (20 if full else 12), nx * (ny - 2) * nz, pml, nx * nz


def work(case):
    """Per step: each interior cell's 9 fields read for one half-step and 3 or 6 of them read and
    written in each (27 values, and 3 of the medium where it is 3-D); an absorbing-strip cell's
    18 field values and 24 split components read and written; a fault node's friction
    parameters and state.  Each half-step needs what the other has written everywhere around it,
    so a pass of many steps needs this once a step."""
    c = case
    size = 8 if c.get("precision") == "f64" else 4
    extra = 3 if c.get("medium") == "3d" else 0
    nbytes = flops = 0.0
    for _, _, _, interior, pml, nodes in _grids(c):
        nbytes += interior * (27 + extra) * size + pml * (66 + extra) * size + nodes * (22 * size + 80)
        flops += interior * 129.0 + pml * 190.0 + nodes * (600.0 if c.get("law") == "fvw" else 150.0)
    return {"bytes": nbytes * c["steps"], "flops": flops * c["steps"]}


# ---------------------------------------------------------------- the same in 64 bits
class _Wave64:
    """The scheme in double precision with whole-array operations: 4th-order staggered velocity
    and stress updates inside, 2nd order at the row next to the fault, split-field absorbing
    strips, a free surface (or a strip) on top, traction at split nodes on the fault row
    j = nyt.  Arrays are [k, j, i]; indices in comments and ranges are 1-based."""

    C1, C2 = 9.0 / 8.0, -1.0 / 24.0

    def __init__(self, m, medium3d=None):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.m, self.law = m, m["law"]
        self.nx, self.ny, self.nz, self.na = m["nxt"], m["nyt"], m["nzt"], m["nabc"]
        self.full = bool(m.get("fspace"))
        self.ks = self.nz - m["nfs"]
        self.dt, self.dh, self.damp = m["dt"], m["dh"], m["damp_s"]
        if medium3d is None:
            shape = (self.nz, self.ny, self.nx)
            self.lam, self.mu, self.d = (self._t(a).view(-1, 1, 1).expand(shape) for a in m["medium"])
        else:
            self.lam, self.mu, self.d = (self._t(a.T) for a in medium3d)
        self.f = {n: torch.zeros((self.nz, self.ny, self.nx), dtype=torch.float64, device=self.dev)
                  for n in ("u", "v", "w", "xx", "yy", "zz", "xy", "yz", "xz")}
        self._strips()
        self._fault()
        self.it = 0

    def _t(self, a):
        return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=self.dev)

    # a[k, j, i] over a box of 1-based inclusive ranges, shifted
    @staticmethod
    def at(a, box, k=0, j=0, i=0):
        (k0, k1), (j0, j1), (i0, i1) = box
        return a[k0 - 1 + k:k1 + k, j0 - 1 + j:j1 + j, i0 - 1 + i:i1 + i]

    def d4(self, a, box, axis, ahead):
        """4th-order difference along an axis: ahead 1: from here to the next point, 0: from the
        previous one to here."""
        s = lambda o: self.at(a, box, **{axis: o + ahead})  # noqa: E731
        return self.C1 * (s(0) - s(-1)) + self.C2 * (s(1) - s(-2))

    def d2(self, a, box, axis, ahead):
        return self.at(a, box, **{axis: ahead}) - self.at(a, box, **{axis: ahead - 1})

    def _strips(self):
        na, nx, ny, ks, n = self.na, self.nx, self.ny, self.ks, self.na - 1
        top = self.m["pml_fact"] * self.m["pml_vp"] / (2.0 * self.dh * n)
        r = torch.arange(1, n + 1, dtype=torch.float64)
        om, half = (0.5 * self.dt * top * ((r - o) / n) ** 4 for o in (0.0, 0.5))
        lo, lo_h = om.flip(0), half.flip(0)

        def prof(count, low=None, high=None):
            p = torch.zeros(count, dtype=torch.float64)
            if low is not None:
                p[:n] = low
            if high is not None:
                p[count - n:] = high
            return p

        boxes = [((na + 1, ks), (na + 1, ny - 1), (2, na)), ((na + 1, ks), (na + 1, ny - 1), (nx - na + 1, nx - 1)),
                 ((na + 1, ks), (2, na), (2, nx - 1)), ((2, na), (2, ny - 1), (2, nx - 1))]
        if self.full:
            boxes.append(((self.nz - na + 1, self.nz - 1), (2, ny - 1), (2, nx - 1)))
        self.strips = []
        for s, (K, J, I) in enumerate(boxes):
            Ju = J if s == 2 else (J[0], J[1] + 1)  # u, w, xz and the normal stresses reach the fault row
            nk, nj, ni = K[1] - K[0] + 1, Ju[1] - Ju[0] + 1, I[1] - I[0] + 1
            x_low, x_high = s != 1, s != 0
            hi, hi_h = (half, om) if s < 2 else (half.flip(0), om.flip(0))  # (so in the scheme's edge strips)
            ox = prof(ni, lo if x_low else None, hi if x_high else None)
            oxs = prof(ni, lo_h if x_low else None, hi_h if x_high else None)
            oy = oys = torch.zeros(nj, dtype=torch.float64)
            if s >= 2:
                oy, oys = prof(nj, lo), prof(nj, lo_h)
            oz = ozs = torch.zeros(nk, dtype=torch.float64)
            if s == 3:
                oz, ozs = prof(nk, lo), prof(nk, lo_h)
            if s == 4:
                oz, ozs = half.clone(), om.clone()
            shape = dict(x=(1, 1, -1), y=(1, -1, 1), z=(-1, 1, 1))
            o = {k: v.to(self.dev).view(shape[k[0]]) for k, v in dict(x=ox, xs=oxs, y=oy, ys=oys, z=oz, zs=ozs).items()}
            zero = lambda rows: torch.zeros((nk, rows, ni), dtype=torch.float64, device=self.dev)  # noqa: E731
            nv = J[1] - J[0] + 1
            a = {c: zero(nj) for c in ("u0", "u1", "u2", "w0", "w1", "w2", "xx0", "xx1", "xx2", "yy0", "yy1", "yy2",
                                       "zz0", "zz1", "zz2", "xz0", "xz1")}
            a.update({c: zero(nv) for c in ("v0", "v1", "v2", "xy0", "xy1", "yz0", "yz1")})
            self.strips.append(dict(u=(K, Ju, I), v=(K, J, I), o=o, a=a, nv=nv, clear=s <= 2 and not self.full))

    def _split(self, st, comp, om, inc):
        o, a = st["o"][om], st["a"][comp]
        if om[0] == "y":
            o = o[:, :a.shape[1], :]
        a.mul_(1.0 - o).add_(inc).div_(1.0 + o)
        return a

    def _fault(self):
        q, fl = {}, self.m["fault"]
        plane = lambda v=0.0: torch.full((self.nz, self.nx), v, dtype=torch.float64, device=self.dev)  # noqa: E731
        up = lambda k: self._t(np.asarray(fl[k]).T)  # noqa: E731
        for n in ("tx", "tz", "RFx", "RFz", "avdx", "avdz", "au", "av", "aw", "uZ", "wX", "distX", "distZ", "slipX",
                  "slipZ", "rise"):
            q[n] = plane()
        q["ruptime"], q["sliptime"] = plane(1e4), plane(1e4)
        q["tabsX"], q["tabsZ"] = plane(1.0 if self.law == "fvw" else 0.0), plane(1.0 if self.law == "fvw" else 0.0)

        def mean4(a):
            b = plane()
            b[1:-1, 1:-1] = (a[1:-1, 1:-1] + a[1:-1, :-2] + a[:-2, 1:-1] + a[:-2, :-2]) / 4
            return b

        q["T0X"], q["T0Z"], q["Dc"] = mean4(up("striniX")), up("striniZ"), up("Dc")
        q["T0X0"] = q["T0X"].clone()
        if self.law == "fvw":
            for n in ("a", "b", "psi", "vw", "fw"):
                q[n + "Z"] = up(n if n != "fw" else "fwZ")
                q[n + "X"] = up(n + "X")
            self.s = {n: float(fl[n]) for n in ("Sn", "v0", "f0", "uini", "wini", "hx0", "hz0", "perturb", "RR2",
                                                "TT2")}
        else:
            q["peakZ"], q["dynZ"], q["coh"] = up("peak_xz"), up("dyn_xz"), up("coh")
            q["peakX"], q["dynX"], q["DcX"] = mean4(q["peakZ"]), mean4(q["dynZ"]), mean4(q["Dc"])
        self.q = q

    # fault-plane values [k, i] of the interior rows, shifted
    def p2(self, a, k=0, i=0):
        return a[self.na + k:self.ks + k, self.na + i:self.nx - self.na + i]

    def row(self, name, k=0, i=0, j=0):
        """A field on the fault row (j = nyt + j)."""
        return self.p2((self.f[name] if isinstance(name, str) else name)[:, self.ny - 1 + j, :], k, i)

    def _newton(self, vt, cd, uw, psi, a):
        e = self.s["v0"] * torch.exp(-psi / a)
        for _ in range(200):
            step = (vt + cd * uw + torch.sinh(uw) * e) / (cd + torch.cosh(uw) * e)
            uw = uw - step
            if float(step.abs().max()) <= 1e-10:
                break
        return uw

    def _velocity(self):
        f, q, at, dth = self.f, self.q, self.at, self.dt / self.dh
        na, ny = self.na, self.ny
        K, I = (na + 1, self.ks), (na + 1, self.nx - na)
        new = {}
        box = (K, (na + 1, ny - 2), I)
        r = dth / at(self.d, box)
        new["u"] = r * (self.d4(f["xx"], box, "i", 0) + self.d4(f["xy"], box, "j", 0) + self.d4(f["xz"], box, "k", 0))
        new["v"] = r * (self.d4(f["xy"], box, "i", 1) + self.d4(f["yy"], box, "j", 1) + self.d4(f["yz"], box, "k", 0))
        new["w"] = r * (self.d4(f["xz"], box, "i", 1) + self.d4(f["yz"], box, "j", 0) + self.d4(f["zz"], box, "k", 1))
        for n in "uvw":
            at(f[n], box).add_(new[n])
        # the row next to the fault
        box = (K, (ny - 1, ny - 1), I)
        r = dth / at(self.d, box)[:, 0]
        inc = dict(u=self.d2(f["xx"], box, "i", 0) + self.d2(f["xy"], box, "j", 0) + self.d2(f["xz"], box, "k", 0),
                   v=self.d2(f["xy"], box, "i", 1) + self.d2(f["yy"], box, "j", 1) + self.d2(f["yz"], box, "k", 0),
                   w=self.d2(f["xz"], box, "i", 1) + self.d2(f["yz"], box, "j", 0) + self.d2(f["zz"], box, "k", 1))
        for n in "uvw":
            g, mem = inc[n][:, 0], self.p2(q["a" + n])
            at(f[n], box)[:, 0].add_(r * (g + self.damp * (g - mem)))
            mem.copy_(g)
        f["v"][:, ny - 1] = f["v"][:, ny - 2]
        # the fault row
        u, w = self.row("u"), self.row("w")
        r = dth / self.row(self.d)
        if self.law != "fvw":
            u.add_(r * 2.0 * (self.p2(q["tx"]) + self.p2(q["RFx"])))
            w.add_(r * 2.0 * (self.p2(q["tz"]) + self.p2(q["RFz"])))
        else:
            s, p2 = self.s, self.p2
            sq = lambda x, y: torch.sqrt(x * x + y * y)  # noqa: E731
            a, psi, wX = p2(q["aX"]), p2(q["psiX"]), p2(q["wX"])
            sr = sq(2 * (wX.abs() + abs(s["wini"])), 2 * (u.abs() + abs(s["uini"])))
            rf = (p2(q["RFz"]) + p2(q["RFz"], 0, -1) + p2(q["RFz"], -1) + p2(q["RFz"], -1, -1)) / 4
            vt = -sq(wX + 2 * r * (rf - p2(q["T0Z"])), u + 2 * r * (p2(q["RFx"]) - p2(q["T0X"])))
            uw = self._newton(vt, 2 * r * s["Sn"] * a, torch.asinh(torch.exp(psi / a) * sr / (2 * s["v0"])), psi, a)
            rate = -torch.sinh(uw) * s["v0"] * torch.exp(-psi / a)
            un = (p2(q["tx"]) + p2(q["T0X"])) * rate / p2(q["tabsX"]) + s["uini"]
            a, psi, uZ = p2(q["aZ"]), p2(q["psiZ"]), p2(q["uZ"])
            sr = sq(2 * (w - s["wini"]), 2 * (uZ - s["uini"]))
            four = lambda x: (p2(x) + p2(x, 0, 1) + p2(x, 1) + p2(x, 1, 1)) / 4  # noqa: E731
            vt = -sq(w + 2 * r * (p2(q["RFz"]) - p2(q["T0Z"])), uZ + 2 * r * (four(q["RFx"]) - four(q["T0X"])))
            uw = self._newton(vt, 2 * r * s["Sn"] * a, torch.asinh(torch.exp(psi / a) * sr / (2 * s["v0"])), psi, a)
            rate = -torch.sinh(uw) * s["v0"] * torch.exp(-psi / a)
            wn = (p2(q["tz"]) + p2(q["T0Z"])) * rate / p2(q["tabsZ"]) + s["wini"]
            u.copy_(un)
            w.copy_(wn)
        for st in self.strips:
            b = st["u"]
            r = self.dt / at(self.d, b) / self.dh
            sp = lambda c, om, x: self._split(st, c, om, x)  # noqa: E731
            at(f["u"], b).copy_(sp("u0", "x", r * self.d2(f["xx"], b, "i", 0)) +
                                sp("u1", "y", r * self.d2(f["xy"], b, "j", 0)) +
                                sp("u2", "z", r * self.d2(f["xz"], b, "k", 0)))
            at(f["w"], b).copy_(sp("w0", "xs", r * self.d2(f["xz"], b, "i", 1)) +
                                sp("w1", "y", r * self.d2(f["yz"], b, "j", 0)) +
                                sp("w2", "z", r * self.d2(f["zz"], b, "k", 1)))
            b = st["v"]
            r = r[:, :st["nv"]]
            at(f["v"], b).copy_(sp("v0", "xs", r * self.d2(f["xy"], b, "i", 1)) +
                                sp("v1", "y", r * self.d2(f["yy"], b, "j", 1)) +
                                sp("v2", "z", r * self.d2(f["yz"], b, "k", 0)))
        if self.full:
            return
        # velocities of the ghost row above the free surface
        n = self.ks - 1
        u, v, w = f["u"], f["v"], f["w"]
        u[n + 1, :, 1:-1] = u[n, :, 1:-1] - (w[n, :, 1:-1] - w[n, :, :-2])
        v[n + 1, 1:-1, 1:-1] = v[n, 1:-1, 1:-1] - (w[n, 2:, 1:-1] - w[n, 1:-1, 1:-1])
        lam, mu = self.lam[n + 1, 1:, 1:-2], self.mu[n + 1, 1:, 1:-2]
        w[n + 1, 1:, 1:-2] = w[n - 1, 1:, 1:-2] - 2 * lam / (lam + 2 * mu) * sum(
            u[k, 1:, 2:-1] - u[k, 1:, 1:-2] + v[k, 1:, 1:-2] - v[k, :-1, 1:-2] for k in (n, n + 1))

    def _stress(self):
        f, at, dth = self.f, self.at, self.dt / self.dh
        na, ny = self.na, self.ny
        u, v, w = f["u"], f["v"], f["w"]
        K, I = (na + 1, self.ks), (na + 1, self.nx - na)
        for box, D in (((K, (na + 1, ny - 2), I), self.d4), ((K, (ny - 1, ny - 1), I), self.d2)):
            lam, mu = at(self.lam, box), at(self.mu, box)
            ex, ey, ez = D(u, box, "i", 1), D(v, box, "j", 0), D(w, box, "k", 0)
            tr = lam * (ex + ey + ez)
            for n, e in (("xx", ex), ("yy", ey), ("zz", ez)):
                at(f[n], box).add_(dth * (tr + 2 * mu * e))
            at(f["xy"], box).add_(dth * 0.5 * (mu + at(self.mu, box, j=1)) * (D(u, box, "j", 1) + D(v, box, "i", 0)))
            at(f["xz"], box).add_(dth * 0.5 * (mu + at(self.mu, box, k=1)) * (D(u, box, "k", 1) + D(w, box, "i", 0)))
            g = dth * 0.5 * (mu + at(self.mu, box, k=1, j=1, i=1))
            at(f["yz"], box).add_(g * (D(v, box, "k", 1) + D(w, box, "j", 1)))
        f["xy"][:, ny - 1] = f["xy"][:, ny - 2]
        f["yz"][:, ny - 1] = f["yz"][:, ny - 2]
        # the fault row
        b = (K, (ny, ny), I)
        lam, mu = at(self.lam, b), at(self.mu, b)
        at(f["xz"], b).add_(dth * 0.5 * (mu + at(self.mu, b, k=1)) * (self.d4(u, b, "k", 1) + self.d4(w, b, "i", 0)))
        ex, ez = self.d4(u, b, "i", 1), self.d4(w, b, "k", 0)
        ey = -lam * (ex + ez) / (lam + 2 * mu)  # twice the jump of v that leaves yy as the row next to it has it
        tr = lam * (ex + ey + ez)
        for n, e in (("xx", ex), ("yy", ey), ("zz", ez)):
            at(f[n], b).add_(dth * (tr + 2 * mu * e))
        r = self.dt / self.dh
        for st in self.strips:
            sp = lambda c, om, x: self._split(st, c, om, x)  # noqa: E731
            b = st["u"]
            lam, mu = at(self.lam, b), at(self.mu, b)
            ex, ey, ez = r * self.d2(u, b, "i", 1), r * self.d2(v, b, "j", 0), r * self.d2(w, b, "k", 0)
            for n in ("xx", "yy", "zz"):
                at(f[n], b).copy_(sp(n + "0", "xs", ex * (lam + 2 * mu if n == "xx" else lam)) +
                                  sp(n + "1", "y", ey * (lam + 2 * mu if n == "yy" else lam)) +
                                  sp(n + "2", "z", ez * (lam + 2 * mu if n == "zz" else lam)))
            g = r * (mu + at(self.mu, b, k=1)) / 2
            at(f["xz"], b).copy_(sp("xz0", "zs", g * self.d2(u, b, "k", 1)) + sp("xz1", "x", g * self.d2(w, b, "i", 0)))
            b = st["v"]
            mu = at(self.mu, b)
            g = r * (mu + at(self.mu, b, j=1)) / 2
            at(f["xy"], b).copy_(sp("xy0", "ys", g * self.d2(u, b, "j", 1)) + sp("xy1", "x", g * self.d2(v, b, "i", 0)))
            g = r * (mu + at(self.mu, b, k=1, j=1, i=1)) / 2
            at(f["yz"], b).copy_(sp("yz0", "zs", g * self.d2(v, b, "k", 1)) +
                                 sp("yz1", "ys", g * self.d2(w, b, "j", 1)))
            if st["clear"]:
                for n in ("xz0", "xz1", "yz0", "yz1"):
                    st["a"][n][-1] = 0
        if not self.full:  # stresses above the free surface
            n = self.ks - 1
            for s in ("zz", "xz", "yz"):
                f[s][n + 1] = -f[s][n if s == "zz" else n - 1]
                f[s][n + 2] = -f[s][n - 1 if s == "zz" else n - 2]
            f["xz"][n] = 0
            f["yz"][n] = 0

    def _boundary(self):
        """Traction, friction, slip and rupture time on the fault; the history planes."""
        f, q, p2, row = self.f, self.q, self.p2, self.row
        d4 = lambda n, ax, ahead: self.C1 * (row(n, **{ax: ahead}) - row(n, **{ax: ahead - 1})) + \
            self.C2 * (row(n, **{ax: ahead + 1}) - row(n, **{ax: ahead - 2}))  # noqa: E731
        pz = (d4("xz", "i", 1) + d4("zz", "k", 1)) / 2 - row("yz", j=-1)
        half = torch.ones((pz.shape[0], 1), dtype=torch.float64, device=self.dev)
        if not self.full:
            pz[-1] = ((row("xz", -1, 1) - row("xz", -1)) / 8 + (row("zz", 1) - row("zz")) / 4 -
                      row("yz", -1, j=-1) / 4)[-1]
            half[-1] = 0.5
        px = (d4("xx", "i", 0) + d4("xz", "k", 0)) / 2 - row("xy", j=-1)
        u, w, imp = row("u"), row("w"), 0.5 * row(self.d) * self.dh / self.dt
        for p, av, rf, t, vel in ((pz, "avdz", "RFz", "tz", w * half), (px, "avdx", "RFx", "tx", u)):
            p2(q[rf]).copy_(p + self.damp * (p - p2(q[av])))
            p2(q[av]).copy_(p)
            p2(q[t]).copy_(-p2(q[rf]) - imp * vel)
        if not self.full:
            inner = slice(self.na, self.nx - self.na)
            q["tx"][self.ks, inner] = q["tx"][self.ks - 1, inner]
            q["tz"][self.ks, inner] = -q["tz"][self.ks - 2, inner]
        X, Z = q["tx"] + q["T0X"], q["tz"] + q["T0Z"]
        avg = lambda a, s: (p2(a) + p2(a, 0, s) + p2(a, s) + p2(a, s, s)) / 4  # noqa: E731
        norm = lambda x, y: torch.sqrt(x * x + y * y)  # noqa: E731
        p2(q["tabsZ"]).copy_(norm(avg(X, 1), p2(Z)))
        p2(q["tabsX"]).copy_(norm(p2(X), avg(Z, -1)))
        four = lambda n, s: (row(n) + row(n, 0, s) + row(n, s) + row(n, s, s)) / 4  # noqa: E731
        uZ, wX = four("u", 1), four("w", -1)
        p2(q["uZ"]).copy_(uZ)
        p2(q["wX"]).copy_(wX)
        time, dt = self.it * self.dt, self.dt
        out = []
        for n, speed, slip, va, vb in (("Z", norm(w, uZ), "distZ", w, uZ), ("X", norm(wX, u), "distX", wX, u)):
            dist = p2(q[slip])
            if self.law == "fvw":
                s, a = self.s, p2(q["a" + n])
                sr = norm(2 * (va.abs() + abs(s["wini"])), 2 * (vb.abs() + abs(s["uini"])))
                fw = p2(q["fw" + n])
                flv = s["f0"] - (p2(q["b" + n]) - a) * torch.log(sr / s["v0"])
                fss = fw + (flv - fw) / (1 + (sr / p2(q["vw" + n])) ** 8) ** 0.125
                pss = a * (torch.log(torch.sinh(fss / a)) + torch.log(2 * s["v0"] / sr))
                psi = p2(q["psi" + n])
                psi.copy_((psi - pss) * torch.exp(-sr * dt / p2(q["Dc"])) + pss)
                out.append(s["Sn"] * a * torch.asinh(sr * torch.exp(psi / a) / (2 * s["v0"])))
                dist.add_(2 * speed * dt)
                moving = 2 * speed > 1e-3
            else:
                dc = p2(q["Dc"] if n == "Z" else q["DcX"])
                weak = p2(q["peak" + n]) * (1 - dist / dc) + p2(q["dyn" + n]) * dist / dc + p2(q["coh"])
                weak = torch.where(dist <= p2(q["Dc"]), weak, p2(q["dyn" + n]) + p2(q["coh"]))
                size = p2(q["tabs" + n])
                slips = size >= weak
                t, t0 = p2(q["t" + n.lower()]), p2(q["T0" + n])
                t.copy_(torch.where(slips, (t + t0) * weak / size - t0, t))
                dist.add_(torch.where(slips, 2 * speed * dt, 0.0 * speed))
                moving = slips & (2 * speed > 1e-3)
            if n == "Z":
                rt = p2(q["ruptime"])
                begun = rt != 1e4
                p2(q["rise"])[moving & begun] = time
                rt[moving & ~begun] = time
                p2(q["slipZ"]).sub_(2 * w * dt)
                p2(q["slipX"]).sub_(2 * uZ * dt)
                st = p2(q["sliptime"])
                st[(st == 1e4) & (dist > p2(q["Dc"]))] = time
        rate_x = -2 * four("u", 1)
        if not self.full:
            rate_x[-1] = (-2 * (row("u") + row("u", 0, 1)) / (4 if self.law == "fvw" else 2))[-1]
        elif self.law == "fvw":
            rate_x[-1] = (-2 * (row("u") + row("u", 0, 1)) / 4)[-1]
        else:
            rate_x[-1] = (-(row("u") + row("u", 0, 1)))[-1]
        if self.law == "fvw":
            planes = [rate_x, -2 * w, out[1], out[0], p2(q["psiZ"]).clone()]
        else:
            X, Z = q["tx"] + q["T0X"], q["tz"] + q["T0Z"]
            sx = avg(X, 1)
            sx[-1] = ((p2(X) + p2(X, 0, 1)) / 2)[-1]
            planes = [rate_x, -2 * w, sx, p2(Z).clone()]
        self.planes = planes
        if self.law == "fvw" and self.m["fault"].get("nucleation"):
            s, th = self.s, time - dt / 2
            if th <= s["TT2"]:
                gt = math.exp((th - s["TT2"]) ** 2 / (th * (th - 2 * s["TT2"]))) if th < s["TT2"] else 1.0
                k = torch.arange(self.na - 1, self.ks + 1, dtype=torch.float64, device=self.dev).view(-1, 1)
                i = torch.arange(self.na - 1, self.nx - self.na + 1, dtype=torch.float64, device=self.dev).view(1, -1)
                rr = (i * self.dh - s["hx0"]) ** 2 + (k * self.dh - s["hz0"]) ** 2
                bump = torch.where(rr < s["RR2"] - self.dh, torch.exp(rr / (rr - s["RR2"] - self.dh)), 0.0 * rr)
                part = (slice(self.na - 2, self.ks), slice(self.na - 2, self.nx - self.na))
                q["T0X"][part] = q["T0X0"][part] + s["perturb"] * bump * gt

    def run(self, steps, stride):
        """The history planes and seismograms of every stride-th step."""
        recs, seis = [], []
        for _ in range(steps):
            self.it += 1
            self._velocity()
            self._stress()
            self._boundary()
            if self.it % stride == 0:
                recs.append([p.cpu().numpy() for p in self.planes])
                seis.append([[float(self.f[n][z - 1, y - 1, x - 1]) for n in "uvw"] for x, y, z in self.m["stations"]])
        out = {n: np.stack([r[h] for r in recs]) for h, n in enumerate(HISTORIES[:len(self.planes)])} if recs else {}
        return out, np.array(seis)

    def final(self):
        out = {n: self.q[n].cpu().numpy().T for n in FINALS}
        out["rise"] = out["rise"] - out["ruptime"]  # the rise time
        return out


def exact(case, seed):
    c = case
    if c["kind"] in ("batch", "serve"):
        n = c.get("models", c.get("requests"))
        if n * c["steps"] > 3000:  # about 6 ms a model and step: beyond 20 s
            return None
        finals = []
        for m in _mixed(c, seed, n):
            w = _Wave64(m)
            w.run(c["steps"], c["steps"] + 1)
            finals.append(w.final())
        return _joined(finals)
    m = _model(c, seed)
    w = _Wave64(m, _medium3d(m, seed) if c["medium"] == "3d" else None)
    out, seis = w.run(c["steps"], c["stride"])
    if c["kind"] == "once":
        return w.final()
    # where the waves have not come to the stations, velocities are below what 32 bits hold
    out["stations"] = seis if c["whole"] and np.abs(seis).max() > 1e-20 else None
    if c["whole"]:
        out.update(w.final())
    return out
