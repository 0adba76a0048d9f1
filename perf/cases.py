"""Performance cases: the work a user of the solver has it do, through its Python binding.

A case is a plain dict. Its "kind" says which entry points it goes through:
  solve  a cavity advanced by a fixed number of outer iterations from given fields: Solver.upload of
         u, v, p, Solver.run, Solver.download of u, v, p into pinned host buffers;
  batch  independent cavities of uneven size advanced in one launch: Batch.run, Batch.results and
         every cavity's u, v, p;
  infer  the warm-start network on one image: Cnn.forward;
  train  one training step of the network on a batch of pairs: Cnn.train_step, Cnn.params.
Fixed work: error_tolerance is 0, so a run does exactly the iterations asked for.
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch
import torch.nn.functional as F

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "simple-hpc_b200"))
import sgpu  # noqa: E402

WEIGHTS = os.path.join(_ROOT, "simple-hpc_b200", "weights", "unet16_l4_cavity.bin")
CHANNELS = (16, 32, 64, 128)  # of the network in WEIGHTS


def _solve(name, nx, ny, iters, pressure="mg", precision="fp64", scheme="QUICK", order=4, re=1000.0, mode="fixed"):
    return ({"name": name} if name else {}) | {"kind": "solve", "nx": nx, "ny": ny, "iters": iters, "pressure": pressure,
            "precision": precision, "scheme": scheme, "order": order, "re": re, "mode": mode}


def listed():
    return [
        # The smallest cavity the repository is configured for (Re 100, 2nd order): every phase is a
        # handful of blocks, so launches, barriers and serial chains are all there is.
        _solve("fp64_mg_32", 32, 32, 20, order=2, re=100.0),
        # The published 128^2 validation case in mixed precision: a run to 1e-5 takes thousands of
        # latency-bound iterations.
        _solve("mixed_mg_128", 128, 128, 200, precision="mixed"),
        # The FP64 method on one GPU at 1024^2, QUICK / 4th order, one V(2,2) cycle per iteration.
        _solve("fp64_mg_1024", 1024, 1024, 60),
        # The plain FP64 arm of the headline benchmark.
        _solve("fp64_mg_4096", 4096, 4096, 24),
        # The headline benchmark: 4096^2, mixed precision.
        _solve("mixed_mg_4096", 4096, 4096, 60, precision="mixed"),
        # A rectangular grid whose sizes are no powers of two: the coarsest level stays at 75 x 125 cells.
        _solve("mixed_mg_600x1000", 600, 1000, 10, precision="mixed"),
        # The one solver pair that the reference's own GPU backend has, on an odd, ragged grid.
        _solve("fp64_redblack_1531x2047", 1531, 2047, 30, pressure="gs_redblack"),
        # Conjugate gradients for p' to the default 1e-6 of ||b||, first-order upwind.
        _solve("fp64_cg_512", 512, 512, 2, pressure="cg", scheme="UDS", order=2),
        # Tolerance-driven p' solves (V-cycles to 1e-5 in FP64 defect correction), as the evaluation of
        # the learned warm start and the generation of its training pairs run them.
        _solve("mixed_mgtol_1024", 1024, 1024, 6, precision="mixed", re=2000.0, mode="tolerance"),
        # A sweep over sizes and Reynolds numbers in one launch.
        {"name": "batch_20", "kind": "batch", "count": 20, "nmin": 64, "nmax": 512, "draw": 7, "iters": 100,
         "precision": "mixed"},
        # Inference of the warm-start network at the level size it runs on inside a solve.
        {"name": "cnn_infer_256", "kind": "infer", "n": 1, "h": 256, "w": 256},
        # Training of the network: batches of 8 pairs on 256^2 levels.
        {"name": "cnn_train_8x256", "kind": "train", "n": 8, "h": 256, "w": 256},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random):
    kind = rng.choices(["mg", "redblack", "cg", "tolerance", "batch", "infer", "train"],
                       [10, 4, 2, 2, 2, 1, 2])[0]
    scheme, order = rng.choice([("QUICK", 4), ("QUICK", 4), ("QUICK", 2), ("UDS", 2)])
    re = round(_log(rng, 100, 5000), 1)

    def level_size(top):
        # coarsest sizes 4..20 of either parity, halved up as far as the case's size goes
        n = int(round(_log(rng, 32, top)))
        k = max(0, int(math.log2(n / rng.uniform(4.5, 20))))
        return max(4, n >> k) << k

    def pair(top):
        nx = level_size(top)
        if rng.random() < 0.5:
            return nx, nx
        m = nx
        while m % 2 == 0 and m // 2 >= 4:
            m //= 2
        k = int(round(math.log2(nx / m)))
        return nx, min(top, max(4, int(round(m * rng.uniform(0.6, 1.6))))) << k if m << k <= top else nx

    def count(cells, budget):  # outer iterations
        return max(2, min(50, int(budget / cells)))

    if kind == "mg":
        precision = rng.choice(["fp64", "mixed"])
        nx, ny = pair(2900)
        return _solve("", nx, ny, count(nx * ny, 1e8), precision=precision, scheme=scheme, order=order, re=re)
    if kind == "redblack":
        nx, ny = int(_log(rng, 24, 2900)), int(_log(rng, 24, 2900))
        return _solve("", nx, ny, count(nx * ny, 1e8), pressure="gs_redblack", scheme=scheme, order=order, re=re)
    if kind == "cg":
        nx, ny = int(_log(rng, 40, 700)), int(_log(rng, 40, 700))
        return _solve("", nx, ny, 2, pressure="cg", scheme=scheme, order=order, re=re)
    if kind == "tolerance":
        nx, ny = pair(2048)
        return _solve("", nx, ny, 4, precision=rng.choice(["fp64", "mixed"]), scheme=scheme, order=order, re=re,
                      mode="tolerance")
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(3, 20), "nmin": 32, "nmax": rng.choice([128, 256, 512]),
                "draw": rng.randrange(1 << 20), "iters": rng.randint(20, 80),
                "precision": rng.choice(["mixed", "mixed", "fp64"])}
    h, w = 8 * rng.randint(4, 32), 8 * rng.randint(4, 32)
    return {"kind": kind, "n": 1 if kind == "infer" else rng.choice([1, 2, 4, 8]), "h": h, "w": w}


# ---- inputs ----

def _config(nx, ny, re, scheme, order, pressure, precision, mode):
    keys = {"N_cells_x": nx, "N_cells_y": ny, "Re": repr(float(re)), "convection_scheme": scheme,
            "diffusion_order": order, "momentum_solver": "gs_multicolour", "pressure_solver": pressure,
            "error_tolerance": 0, "maxit": 1000000, "backend": "gpu", "precision": precision, "mg_mode": mode}
    if mode == "tolerance":
        keys.update(pressure_tolerance="1e-5", pressure_maxit=100)
    return "".join(f"{k} = {v}\n" for k, v in keys.items())


def _params(case):
    return sgpu.params_from_config(_config(case["nx"], case["ny"], case["re"], case["scheme"], case["order"],
                                           case["pressure"], case["precision"], case["mode"]))


def _fields(nx, ny, h, seed):
    """u, v, p of a developing flow: the lid's shear layer, a few smooth vortices and a pressure of
    their size, in the solver's full-grid layout (walls and ghost cells zero)."""
    r = random.Random(seed)
    dev = "cuda"
    y = (torch.arange(nx, device=dev, dtype=torch.float64) + 0.5) / nx  # distance from the lid
    x = (torch.arange(ny, device=dev, dtype=torch.float64) + 0.5) / ny
    u = torch.zeros((nx + 2 * h + 1, ny + 2 * h + 1), device=dev, dtype=torch.float64)
    v, p = torch.zeros_like(u), torch.zeros_like(u)
    xw, yw = x + 0.5 / ny, y - 0.5 / nx  # where u and v sit
    ui = torch.outer(torch.exp(-y * r.uniform(8, 20)), torch.sin(math.pi * xw).clamp_min(0.0) ** 0.5 * 0.6)
    vi = torch.zeros_like(ui)
    pi = torch.zeros_like(ui)
    for _ in range(4):
        a, m, n = r.uniform(-0.1, 0.1), r.randint(1, 3), r.randint(1, 3)
        s2 = lambda t, k: torch.sin(k * math.pi * t) ** 2  # noqa: E731
        s1 = lambda t, k: torch.sin(2 * k * math.pi * t)  # noqa: E731
        ui += torch.outer(s1(y, m), a * s2(xw, n))
        vi += torch.outer(s2(yw, m), a * s1(x, n))
        pi += torch.outer(torch.cos(m * math.pi * y), a * a * torch.cos(n * math.pi * x))
    u[h:h + nx, h + 1:h + ny] = ui[:, :ny - 1]
    v[h + 1:h + nx, h + 1:h + ny + 1] = vi[1:]
    p[h:h + nx, h + 1:h + ny + 1] = pi - pi.mean()
    return u, v, p


def _images(case, seed):
    """Network inputs and targets as the solver writes them: b and AP of a level in units of their
    scale, and a smooth p'."""
    r = np.random.default_rng(seed)
    n, h, w = case["n"], case["h"], case["w"]
    y, x = (np.arange(h) + 0.5) / h, (np.arange(w) + 0.5) / w
    inp = np.empty((n, h, w, 2), np.float32)
    t = np.zeros((n, h, w), np.float32)
    for i in range(n):
        for _ in range(6):
            k, m = r.integers(1, 6, 2)
            t[i] += r.normal() * np.outer(np.cos(k * np.pi * y), np.cos(m * np.pi * x)) / (k * k + m * m)
        b = t[i] * r.uniform(0.5, 2) + 0.3 * r.standard_normal((h, w))
        inp[i, :, :, 0] = b / np.sqrt(np.mean(b * b))
        ap = 1.0 + 0.2 * np.outer(np.exp(-6 * y), np.sin(np.pi * x)) + 0.01 * r.standard_normal((h, w))
        inp[i, :, :, 1] = ap / ap.mean() - 1.0
    return inp, t * np.float32(20.0)


def _cavities(case, seed):
    """The cavities' sizes belong to the case, their Reynolds numbers to the seed."""
    sizes = [n for n in (32, 64, 96, 128, 192, 256, 384, 512) if case["nmin"] <= n <= case["nmax"]]
    ns = random.Random(case["draw"])
    rs = random.Random(seed)
    return [(ns.choice(sizes), round(_log(rs, 100, 5000), 2)) for _ in range(case["count"])]


def _pinned(shape, pool):
    t = torch.empty(shape, dtype=torch.float64, pin_memory=True)
    pool.append(t)
    return t.numpy()


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind}
    if kind == "solve":
        p = _params(case)
        keep = []
        ins, outs = [], []
        for f in _fields(case["nx"], case["ny"], p.H, seed):
            a = _pinned(p.shape, keep)
            a[...] = f.cpu().numpy()
            ins.append(a)
            outs.append(_pinned(p.shape, keep))
        state.update(solver=sgpu.Solver(p), iters=case["iters"], ins=ins, outs=outs, keep=keep)
    elif kind == "batch":
        ps = [sgpu.params_from_config(_config(n, n, re, "QUICK", 2, "mg", case["precision"], "fixed"))
              for n, re in _cavities(case, seed)]
        state.update(batch=sgpu.Batch(ps), iters=case["iters"])
    elif kind == "infer":
        state.update(net=sgpu.Cnn(path=WEIGHTS), x=_images(case, seed)[0])
    else:
        x, t = _images(case, seed)
        state.update(net=sgpu.Cnn(path=WEIGHTS), x=x, t=t)
    return state


def run(state):
    kind = state["kind"]
    if kind == "solve":
        s = state["solver"]
        for f, a in zip((sgpu.F_U, sgpu.F_V, sgpu.F_P), state["ins"]):
            s.upload(f, a)
        _, log = s.run(state["iters"])
        u, v, p = (s.download(f, out=a) for f, a in zip((sgpu.F_U, sgpu.F_V, sgpu.F_P), state["outs"]))
        return {"log": log, "p": p, "u": u, "v": v}
    if kind == "batch":
        b = state["batch"]
        b.run(state["iters"])
        r = b.results()
        out = {"iterations": r["iterations"], "residuals": r["residuals"]}
        for c in range(len(b.params)):
            for name, f in (("u", sgpu.F_U), ("v", sgpu.F_V), ("p", sgpu.F_P)):
                out[f"{c:02d}{name}"] = b.download(c, f)
        return out
    if kind == "infer":
        return state["net"].forward(state["x"])
    loss = state["net"].train_step(state["x"], state["t"], 1e-4)
    return {"loss": loss, "params": state["net"].params()}


# ---- the work a pass cannot do without ----

def _iteration_work(cells):
    # per cell and outer iteration: u, v, p read and one velocity written by each momentum component,
    # u and v read and p' written by the pressure solve, all four read and u, v, p written by the
    # correction; arithmetic of 8 momentum sweeps, 2 assemblies and about 10 passes over p'
    return 144.0 * cells, 700.0 * cells


def work(case):
    kind = case["kind"]
    if kind == "solve":
        cells = case["nx"] * case["ny"]
        b, f = _iteration_work(cells)
        return {"bytes": case["iters"] * b + 6 * 8.0 * cells, "flops": case["iters"] * f}
    if kind == "batch":
        cells = sum(n * n for n, _ in _cavities(case, 0))
        b, f = _iteration_work(cells)
        return {"bytes": case["iters"] * b + 3 * 8.0 * cells, "flops": case["iters"] * f}
    px = case["n"] * case["h"] * case["w"]
    per = 2 * CHANNELS[0]  # the 1x1 head, then two 3x3 convolutions per level, down and up
    for l, c in enumerate(CHANNELS):
        cin = CHANNELS[l - 1] if l else 2
        per += 2 * 9 * (cin * c + c * c) / 4 ** l
        if l + 1 < len(CHANNELS):
            per += 2 * 9 * ((CHANNELS[l + 1] + c) * c + c * c) / 4 ** l
    # training: the convolutions of the input and of the weight gradients, and Adam's arrays
    return ({"bytes": 12.0 * px, "flops": per * px} if kind == "infer" else
            {"bytes": 12.0 * px + 7 * 4 * 489169.0, "flops": 3 * per * px})


# ---- the same results in 64 bits, from the method's definition, in plain torch ----

class _Cavity:
    """SIMPLE on the staggered grid: rows i from the lid down, columns j from west to east, halo h."""

    def __init__(self, case, fields):
        self.c, self.nx, self.ny, self.h = case, case["nx"], case["ny"], 2
        self.dx, self.dy, self.nu = 1.0 / self.ny, 1.0 / self.nx, 1.0 / case["re"]
        self.u, self.v, self.p = fields
        dev = self.u.device
        i = torch.arange(self.u.shape[0], device=dev)[:, None]
        j = torch.arange(self.u.shape[1], device=dev)[None, :]
        h = self.h
        self.ncol = 2 if case["scheme"] == "UDS" and case["order"] == 2 else 5
        colour = (i + j) % 2 if self.ncol == 2 else (i + 3 * j) % 5
        self.ur = (slice(h, h + self.nx), slice(h + 1, h + self.ny))
        self.vr = (slice(h + 1, h + self.nx), slice(h + 1, h + self.ny + 1))
        self.pr = (slice(h, h + self.nx), slice(h + 1, h + self.ny + 1))
        self.colours = {id(r): [(colour == c)[r] for c in range(self.ncol)] for r in (self.ur, self.vr)}
        self.band = (j == h + 1) | (j == self.ny + h) | (i == self.nx + h - 1) | (i == h)

    @staticmethod
    def at(f, r, di, dj):
        return f[r[0].start + di:r[0].stop + di, r[1].start + dj:r[1].stop + dj]

    def coefficients(self, ue, uw, vn, vs, r):
        pos = lambda a: a.clamp_min(0.0)  # noqa: E731
        dx, dy, nu = self.dx, self.dy, self.nu
        band = self.band[r]
        uds = [dy * pos(-ue), dy * pos(uw), dx * pos(-vn), dx * pos(vs)] + [torch.zeros_like(ue)] * 4
        if self.c["scheme"] == "QUICK":
            q = [-dy * (-0.75 * pos(-ue) + 0.375 * pos(ue) - 0.125 * pos(-uw)),
                 -dy * (-0.125 * pos(ue) + 0.375 * pos(-uw) - 0.75 * pos(uw)),
                 -dx * (-0.75 * pos(-vn) + 0.375 * pos(vn) - 0.125 * pos(-vs)),
                 -dx * (-0.125 * pos(vn) + 0.375 * pos(-vn) - 0.75 * pos(vs)),
                 -0.125 * dy * pos(-ue), -0.125 * dy * pos(uw), -0.125 * dx * pos(-vn), -0.125 * dx * pos(vs)]
            conv = [torch.where(band, a, b) for a, b in zip(uds, q)]
        else:
            conv = uds
        e, n = dy * nu / dx, dx * nu / dy
        two = [e, e, n, n, 0.0, 0.0, 0.0, 0.0, 2 * (e + n)]
        four = [4 / 3 * e, 4 / 3 * e, 4 / 3 * n, 4 / 3 * n, -e / 12, -e / 12, -n / 12, -n / 12, 2.5 * (e + n)]
        ap = sum(conv)
        d = two if self.c["order"] == 2 else [torch.where(band, a, b) for a, b in zip(
            torch.tensor(two, device=ue.device, dtype=torch.float64),
            torch.tensor(four, device=ue.device, dtype=torch.float64))]
        return [c + k for c, k in zip(conv, d)], ap + d[8]

    def neighbours(self, k, x, r):
        at = self.at
        s = k[0] * at(x, r, 0, 1) + k[1] * at(x, r, 0, -1) + k[2] * at(x, r, -1, 0) + k[3] * at(x, r, 1, 0)
        if self.ncol == 5:
            s += (k[4] * at(x, r, 0, 2) + k[5] * at(x, r, 0, -2)) + (k[6] * at(x, r, -2, 0) + k[7] * at(x, r, 2, 0))
        return s

    def momentum(self, comp):
        at, h, u, v, p = self.at, self.h, self.u, self.v, self.p
        if comp == "u":
            r, x = self.ur, u
            u[h - 1, h + 1:h + self.ny + 1] = 2 - u[h, h + 1:h + self.ny + 1]
            u[h + self.nx, h + 1:h + self.ny + 1] = -u[h + self.nx - 1, h + 1:h + self.ny + 1]
            faces = [(u[r] + at(u, r, 0, 1)) / 2, (u[r] + at(u, r, 0, -1)) / 2, (v[r] + at(v, r, 0, 1)) / 2,
                     (at(v, r, 1, 0) + at(v, r, 1, 1)) / 2]
            force = (p[r] - at(p, r, 0, 1)) * self.dy
        else:
            r, x = self.vr, v
            v[h:h + self.nx, h] = -v[h:h + self.nx, h + 1]
            v[h:h + self.nx, h + self.ny + 1] = -v[h:h + self.nx, h + self.ny]
            faces = [(at(u, r, -1, 0) + u[r]) / 2, (at(u, r, 0, -1) + at(u, r, -1, -1)) / 2,
                     (v[r] + at(v, r, -1, 0)) / 2, (v[r] + at(v, r, 1, 0)) / 2]
            force = (p[r] - at(p, r, -1, 0)) * self.dx
        k, ap = self.coefficients(*faces, r)
        res = (self.neighbours(k, x, r) + force - ap * x[r]).abs().sum()
        for _ in range(4):
            for mask in self.colours[id(r)]:
                new = 0.3 * (self.neighbours(k, x, r) + force) / ap + 0.7 * x[r]
                x[r] = torch.where(mask, new, x[r])
        full = torch.ones_like(x)
        full[r] = ap
        return full, res

    def iterate(self):
        at, r, dx, dy = self.at, self.pr, self.dx, self.dy
        apu, ru = self.momentum("u")
        apv, rv = self.momentum("v")
        pad = lambda a: F.pad(a, (1, 1, 1, 1))  # noqa: E731
        e, w = dy * dy / apu[r], dy * dy / at(apu, r, 0, -1)
        n, s = dx * dx / apv[r], dx * dx / at(apv, r, 1, 0)
        e[:, -1], w[:, 0], n[0], s[-1] = 0.0, 0.0, 0.0, 0.0
        b = -dx * (self.v[r] - at(self.v, r, 1, 0)) - dy * (self.u[r] - at(self.u, r, 0, -1))
        rp = b.abs().sum()
        q = getattr(self, "solve_" + self.c["pressure"])((e, w, n, s), b)
        q = pad(q)
        i = (slice(1, -1), slice(1, -1))
        du = dy * (q[i] - at(q, (slice(1, 1 + self.nx), slice(1, 1 + self.ny)), 0, 1)) / apu[r]
        dv = dx * (q[i] - at(q, (slice(1, 1 + self.nx), slice(1, 1 + self.ny)), -1, 0)) / apv[r]
        self.u[self.ur] += du[:, :-1]
        self.v[self.vr] += dv[1:]
        self.p[r] += 0.2 * q[i]
        return ru, rv, rp

    # p': links (e, w, n, s), x padded by one cell on each side
    @staticmethod
    def flow(k, x):
        return k[0] * x[1:-1, 2:] + k[1] * x[1:-1, :-2] + k[3] * x[2:, 1:-1] + k[2] * x[:-2, 1:-1]

    @staticmethod
    def checker(b, first):
        i = torch.arange(b.shape[0], device=b.device)[:, None]
        j = torch.arange(b.shape[1], device=b.device)[None, :]
        return ((i + j + first) & 1) == 0

    def smooth(self, k, ap, b, x, sweeps, masks):
        for _ in range(sweeps):
            for m in masks:
                x[1:-1, 1:-1] = torch.where(m, (b + self.flow(k, x)) / ap, x[1:-1, 1:-1])

    def solve_gs_redblack(self, k, b):
        x = F.pad(torch.zeros_like(b), (1, 1, 1, 1))
        start = (self.h + self.h + 1) & 1  # colour of the first cell, counted over the full grid
        self.smooth(k, sum(k), b, x, 8, (self.checker(b, start), self.checker(b, 1 - start)))
        return x[1:-1, 1:-1]

    def solve_cg(self, k, b):
        ap = sum(k)
        b = b - b.mean()
        x, r = torch.zeros_like(b), b.clone()
        z = r / ap
        z -= z.mean()
        d, rz, nb = z.clone(), (r * z).sum(), b.norm()
        for _ in range(1000):
            q = ap * d - self.flow(k, F.pad(d, (1, 1, 1, 1)))
            alpha = rz / (d * q).sum()
            x += alpha * d
            r -= alpha * q
            if r.norm() <= 1e-6 * nb:
                break
            z = r / ap
            z -= z.mean()
            new = (r * z).sum()
            d = z + (new / rz) * d
            rz = new
        return x - x.mean()

    def cycle(self, k, b, x):
        ap = sum(k)
        masks = (self.checker(b, 0), self.checker(b, 1))
        nx, ny = b.shape
        if nx % 2 or ny % 2 or nx // 2 < 4 or ny // 2 < 4:
            b = b - b.mean()
            bn = b.norm()
            for _ in range(200):
                self.smooth(k, ap, b, x, 1, masks)
                if (b - ap * x[1:-1, 1:-1] + self.flow(k, x)).norm() < 1e-10 * bn:
                    break
            x[1:-1, 1:-1] -= x[1:-1, 1:-1].mean()
            return
        self.smooth(k, ap, b, x, 2, masks)
        r = b - ap * x[1:-1, 1:-1] + self.flow(k, x)
        e, w, n, s = k
        coarse = (e[0::2, 1::2] + e[1::2, 1::2], w[0::2, 0::2] + w[1::2, 0::2],
                  n[0::2, 0::2] + n[0::2, 1::2], s[1::2, 0::2] + s[1::2, 1::2])
        rc = r[0::2, 0::2] + r[0::2, 1::2] + r[1::2, 0::2] + r[1::2, 1::2]
        xc = F.pad(torch.zeros_like(rc), (1, 1, 1, 1))
        self.cycle(coarse, rc, xc)
        x[1:-1, 1:-1] += 1.8 * xc[1:-1, 1:-1].repeat_interleave(2, 0).repeat_interleave(2, 1)
        self.smooth(k, ap, b, x, 2, masks)

    def solve_mg(self, k, b):
        b = b - b.mean()
        x = F.pad(torch.zeros_like(b), (1, 1, 1, 1))
        cycles, tol = (100, 1e-5 * b.norm()) if self.c["mode"] == "tolerance" else (1, None)
        total = torch.zeros_like(b)
        ap, rhs = sum(k), b
        for _ in range(cycles):
            self.cycle(k, rhs, x)
            if tol is None:
                return x[1:-1, 1:-1] - x[1:-1, 1:-1].mean()
            if self.c["precision"] == "mixed":  # each cycle solves, from zero, for a correction
                total = total + x[1:-1, 1:-1]
                x = F.pad(total, (1, 1, 1, 1))
            r = b - ap * x[1:-1, 1:-1] + self.flow(k, x)
            if r.norm() <= tol:
                break
            if self.c["precision"] == "mixed":
                rhs, x = r, torch.zeros_like(x)
        return x[1:-1, 1:-1] - x[1:-1, 1:-1].mean()

    def go(self, iters):
        log = []
        for k in range(iters):
            log.append((float(k + 1), *(float(t) for t in self.iterate())))
        return np.array(log)


def _network(case, seed, params, grad):
    """The U-Net in 64 bits from its FP32 parameters (weights rounded to BF16, as it is defined)."""
    dev = "cuda"
    x, t = _images(case, seed)
    w = params.to(dev, torch.float64).requires_grad_(grad)
    h = F.pad(torch.from_numpy(x).to(dev, torch.float64), (0, CHANNELS[0] - 2)).permute(0, 3, 1, 2)
    at = 0

    def conv(a, cout):
        nonlocal at
        cin = a.shape[1]
        k = w[at:at + cout * 9 * cin].reshape(cout, 3, 3, cin).permute(0, 3, 1, 2)
        k = k + (k.detach().to(torch.bfloat16).to(torch.float64) - k.detach())
        at += cout * 9 * cin
        bias = w[at:at + cout]
        at += cout
        cols = F.unfold(a, 3, padding=1) if a[0].numel() * 9 < 1 << 27 else None
        y = torch.matmul(k.reshape(cout, -1), cols) + bias[:, None]
        return F.relu(y.reshape(a.shape[0], cout, a.shape[2], a.shape[3]))

    skips = []
    for l, c in enumerate(CHANNELS):
        if l:
            h = F.avg_pool2d(h, 2)
        h = conv(conv(h, c), c)
        skips.append(h)
    for l in range(len(CHANNELS) - 2, -1, -1):
        h = torch.cat([F.interpolate(h, scale_factor=2, mode="nearest"), skips[l]], 1)
        h = conv(conv(h, CHANNELS[l]), CHANNELS[l])
    out = torch.einsum("nchw,c->nhw", h, w[at:at + CHANNELS[0]]) + w[at + CHANNELS[0]]
    if not grad:
        return out.detach().cpu().numpy()
    loss = ((out - torch.from_numpy(t).to(dev, torch.float64)) ** 2).mean()
    g, = torch.autograd.grad(loss, w)
    # Adam's first step (beta 0.9 and 0.999, eps 1e-8)
    return {"loss": float(loss.detach()), "params": (w - 1e-4 * g / (g.abs() + 1e-8)).detach().cpu().numpy()}


def _weights():
    raw = np.fromfile(WEIGHTS, np.float32, offset=16)  # 16 bytes of header, then the parameters
    return torch.from_numpy(raw)


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        c = _Cavity(case, _fields(case["nx"], case["ny"], 2, seed))
        log = c.go(case["iters"])
        return {"log": log, "p": c.p.cpu().numpy(), "u": c.u.cpu().numpy(), "v": c.v.cpu().numpy()}
    if kind == "batch":
        out = {"iterations": None, "residuals": None}
        # the first two cavities only: all of them would take minutes
        for k, (n, re) in enumerate(_cavities(case, seed)):
            got = None
            if k < 2:
                one = _solve("", n, n, case["iters"], precision=case["precision"], order=2, re=re)
                zero = [torch.zeros((n + 5, n + 5), device="cuda", dtype=torch.float64) for _ in range(3)]
                got = _Cavity(one, zero)
                got.go(case["iters"])
            for f in ("u", "v", "p"):
                out[f"{k:02d}{f}"] = getattr(got, f).cpu().numpy() if got else None
        return out
    return _network(case, seed, _weights(), kind == "train")
