"""The calls a program makes on the wind-tunnel engine, as timed cases.

A case is one pass of a program's loop over the public API (Solver3D, Solver, Batch2D): a chunk of
steps, then the force samples and the macro field, as the validation loops and the pages read them;
a moved obstacle and a few steps (dragging it); one shape gradient. ``prepare`` builds what the
program holds before the call, ``run`` is one pass, ``exact`` evaluates the same pass in 64 bits with
plain torch on index tables of its own.

Force samples are returned in the arithmetic type of the run (float32 except for FP64 storage): the
library adds up, in 64 bits, momentum terms of that type. The shape gradient dJ/dSDF of the FP32
adjoint is returned as float32 for the same reason.
"""
import math

import numpy as np
import torch

from cells_b200 import Batch2D, Solver, Solver3D
from cells_b200._lib import pinned_empty

# ---------------------------------------------------------------------------------------------- cases


def _tunnel3(name, w, h, d, precision, steps, **kw):
    c = {"name": name, "kind": "tunnel3d", "width": w, "height": h, "depth": d, "precision": precision,
         "steps": steps, "body": "sphere", "size": 0.16, "re": 200.0, "smagorinsky": 0.0, "force_every": 1}
    c.update(kw)
    return c


def listed():
    return [
        # one frame of an interactive page on a small grid: a few steps, then the forces and the field
        _tunnel3("frame_64x32x32_fp32", 64, 32, 32, "fp32", 8, re=100.0, size=0.2),
        # the 3D page's body size on its half grid with the subgrid model, FP16 storage, forces every 4 steps
        _tunnel3("wake_128x64x64_fp16_smag", 128, 64, 64, "fp16", 100, size=0.2, smagorinsky=0.1, force_every=4),
        # the headline tunnel (sphere d = 16 at Re 200) in chunks of 400 steps, the validation loop's chunk
        _tunnel3("tunnel_192x96x96_fp32", 192, 96, 96, "fp32", 400, size=1 / 6),
        _tunnel3("tunnel_192x96x96_bf16", 192, 96, 96, "bf16", 400, size=1 / 6),
        # the 64-bit run that storage errors are stated against
        _tunnel3("tunnel_192x96x96_fp64", 192, 96, 96, "fp64", 100, size=1 / 6),
        # the largest configured grid in the two storages that are compared on it
        _tunnel3("tunnel_256x128x128_fp32", 256, 128, 128, "fp32", 200),
        _tunnel3("tunnel_256x128x128_fp16", 256, 128, 128, "fp16", 200),
        # a user's own box: no dimension even, a cube, the subgrid model
        _tunnel3("ragged_161x83x75_fp32_smag", 161, 83, 75, "fp32", 100, body="cube", smagorinsky=0.1),
        # dragging the obstacle on the page: new SDF, eight steps, forces and field
        _tunnel3("drag_192x96x96_fp16", 192, 96, 96, "fp16", 8, kind="moving3d", size=0.2, re=100.0),
        # the 2D cylinder tunnel (Re 100), one chunk of 400 steps with a force sample each step
        {"name": "cylinder_400x100", "kind": "tunnel2d", "width": 400, "height": 100, "precision": "fp32",
         "steps": 400, "mode": "tunnel", "re": 100.0, "smagorinsky": 0.0, "force_every": 1},
        # 64 section tunnels of uneven sizes advanced together, 100 steps (no force sampling)
        {"name": "batch_64_sections", "kind": "batch2d", "tunnels": 64, "width_min": 256, "width_max": 1024,
         "sizes_seed": 7, "steps": 100, "smagorinsky": 0.1, "force_every": 0},
        # one drag gradient of a star-shaped body: set the shape, start the flow, record, sweep back
        {"name": "gradient_128x64x64", "kind": "adjoint3d", "width": 128, "height": 64, "depth": 64, "precision": "fp32",
         "steps": 1000, "window": 400, "every": 100, "re": 150.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tunnel3d"] * 6 + ["moving3d"] + ["tunnel2d"] * 2 + ["batch2d"] + ["adjoint3d"])
    if kind in ("tunnel3d", "moving3d"):
        w = _log_int(rng, 48, 256)
        h = max(20, int(w * rng.uniform(0.4, 0.55)))
        d = max(20, int(w * rng.uniform(0.4, 0.55)))
        if rng.random() < 0.6:  # most programs take even widths; the rest of them none in particular
            w, h, d = w + w % 2, h + h % 2, d + d % 2
        w, h, d = min(w, 256), min(h, 128), min(d, 128)
        precision = rng.choice(["fp32", "fp32", "fp16", "fp16", "bf16", "fp64"])
        if kind == "moving3d":
            steps = rng.randint(4, 16)
        else:
            most = 7e8 / (w * h * d) / {"fp64": 2.5}.get(precision, 1.0)
            steps = max(8, min(_log_int(rng, 8, 400), int(most)))
        c = _tunnel3("", w, h, d, precision, steps, kind=kind, body=rng.choice(["sphere", "cube", "cylinder"]),
                     size=round(rng.uniform(0.14, 0.24), 3), re=round(rng.uniform(60.0, 200.0), 1),
                     smagorinsky=rng.choice([0.0, 0.0, 0.1]), force_every=rng.choice([0, 1, 1, 4]))
        del c["name"]
        return c
    if kind == "tunnel2d":
        mode = rng.choice(["tunnel", "tunnel", "channel", "cavity"])
        w = _log_int(rng, 64, 1024)
        h = max(24, int(w * (1.0 if mode == "cavity" else rng.uniform(0.2, 0.5))))
        steps = max(20, min(_log_int(rng, 50, 1000), int(2e8 / (w * h))))
        return {"kind": kind, "width": w, "height": h, "precision": rng.choice(["fp32", "fp32", "fp64"]), "steps": steps,
                "mode": mode, "re": round(rng.uniform(50.0, 200.0), 1), "smagorinsky": rng.choice([0.0, 0.0, 0.1]),
                "force_every": rng.choice([0, 1, 1, 4])}
    if kind == "batch2d":
        return {"kind": kind, "tunnels": rng.randint(3, 64), "width_min": 128, "width_max": rng.randint(300, 1024),
                "sizes_seed": rng.randint(1, 10 ** 6), "steps": _log_int(rng, 20, 200), "smagorinsky": rng.choice([0.0, 0.1]),
                "force_every": rng.choice([0, 0, 1])}
    w = _log_int(rng, 64, 128)
    return {"kind": kind, "width": w, "height": max(32, w // 2 + rng.randint(-3, 3)), "depth": max(32, w // 2 + rng.randint(-3, 3)),
            "precision": "fp32", "steps": rng.randint(200, 800), "window": rng.randint(50, 150), "every": rng.choice([50, 100]),
            "re": round(rng.uniform(80.0, 150.0), 1)}


# --------------------------------------------------------------------------------------------- inputs

U = 0.1  # inflow speed of every tunnel


def _tau(re, u, length):
    return min(max(3.0 * u * length / re + 0.5, 0.51), 1.0)


def _grid3(c):
    z, y, x = np.meshgrid(np.arange(c["depth"], dtype=np.float64), np.arange(c["height"], dtype=np.float64),
                          np.arange(c["width"], dtype=np.float64), indexing="ij")
    return x, y, z


def _star_terms(nx, ny, nz):
    # the real harmonics of degree <= 3 up to their normalisation, as polynomials of the direction
    return [np.ones_like(nx), ny, nz, nx, nx * ny, ny * nz, 3 * nz * nz - 1, nx * nz, nx * nx - ny * ny,
            ny * (3 * nx * nx - ny * ny), nx * ny * nz, ny * (5 * nz * nz - 1), nz * (5 * nz * nz - 3),
            nx * (5 * nz * nz - 1), nz * (nx * nx - ny * ny), nx * (nx * nx - 3 * ny * ny)]


def _body3(c, rng, shift=0.0):
    """The obstacle's signed distance (float32, negative inside), about (W/4, H/2, D/2) give or take a
    fraction of a cell from the seed, and its reference length."""
    x, y, z = _grid3(c)
    off = rng.uniform(-0.5, 0.5, 3)
    x = x - (c["width"] / 4 + off[0] + shift)
    y = y - (c["height"] / 2 + off[1])
    z = z - (c["depth"] / 2 + off[2])
    if c["kind"] == "adjoint3d":
        r0 = 0.1875 * c["height"]
        r = np.sqrt(x * x + y * y + z * z)
        s = 1.0 / np.maximum(r, 1e-9)
        coef = 0.02 * rng.standard_normal(16)
        radius = r0 * (1 + sum(k * t for k, t in zip(coef, _star_terms(x * s, y * s, z * s))))
        return (r - radius).astype(np.float32).reshape(-1), 2 * r0
    size = c["size"] * c["height"]
    if c["body"] == "sphere":
        d = np.sqrt(x * x + y * y + z * z) - size / 2
    elif c["body"] == "cylinder":
        d = np.sqrt(x * x + y * y) - size / 2
    else:
        q = [np.abs(v) - size / 2 for v in (x, y, z)]
        outside = np.sqrt(sum(np.maximum(v, 0) ** 2 for v in q))
        d = outside + np.minimum(np.maximum(np.maximum(q[0], q[1]), q[2]), 0)
    return d.astype(np.float32).reshape(-1), size


def _macro3(c, rng):
    n = c["width"] * c["height"] * c["depth"]
    m = np.empty((n, 4), dtype=np.float32)
    m[:, :3] = 2e-3 * (rng.random((n, 3), dtype=np.float32) - 0.5)
    m[:, 0] += U
    m[:, 3] = 1.0
    return m.reshape(-1)


def _sizes2(c):
    """(width, height, chord, angle, Re) of each tunnel of a batch: width log-uniform, height a
    quarter of it, chord a fifth of the height."""
    r = np.random.default_rng(c["sizes_seed"])
    out = []
    for _ in range(c["tunnels"]):
        w = int(round(math.exp(r.uniform(math.log(c["width_min"]), math.log(c["width_max"])))))
        h = int(round(w / 4))
        out.append((w, h, h / 5, math.radians(r.uniform(-8, 12)), r.uniform(50, 400)))
    return out


def _section2(w, h, chord, angle, off):
    """A thin rounded section (a capsule of 12% thickness) with its nose ahead of W/4."""
    y, x = np.mgrid[0:h, 0:w].astype(np.float64)
    x0, y0 = w / 4 - chord / 3 + off[0], h / 2 + off[1]
    ex, ey = math.cos(-angle), math.sin(-angle)
    t = np.clip((x - x0) * ex + (y - y0) * ey, 0, chord)
    return (np.hypot(x - x0 - t * ex, y - y0 - t * ey) - 0.06 * chord).astype(np.float32).reshape(-1)


def _macro2(w, h, u, rng):
    m = np.zeros((w * h, 4), dtype=np.float32)
    m[:, 0] = 1.0
    m[:, 1] = u
    m[:, 2] = 2e-3 * (rng.random(w * h, dtype=np.float32) - 0.5)
    return m.reshape(-1)


def _config2(c):
    """Solver config, SDF and start field of a single 2D tunnel: the cylinder tunnel, a channel driven
    by a body force between no-slip walls, or a lid-driven cavity."""
    w, h = c["width"], c["height"]
    if c["mode"] == "tunnel":
        return dict(left=2, right=2, bottom=2, top=2, tau=_tau(c["re"], U, h / 5), spongeFraction=0.15, spongeTau=1.0,
                    absorb=0.02, uIn=U)
    if c["mode"] == "channel":
        tau = 0.8
        return dict(left=0, right=0, bottom=1, top=1, tau=tau, bodyForce=(8 * (tau - 0.5) / 3 * 0.05 / (h * h), 0.0))
    return dict(left=1, right=1, bottom=1, top=3, tau=_tau(c["re"], U, h), uLid=U)


def _inputs(case, seed):
    """What the library is given: configs, SDFs and start fields, from the seed alone."""
    rng = np.random.default_rng(seed)
    k = case["kind"]
    if k in ("tunnel3d", "moving3d", "adjoint3d"):
        state = rng.bit_generator.state
        sdf, length = _body3(case, rng)
        sdfs = [sdf]
        if k == "moving3d":
            for shift in (1.3, 0.0):
                rng.bit_generator.state = state
                sdfs.append(_body3(case, rng, shift)[0])
        cfg = dict(precision=case["precision"], tau=_tau(case["re"], U, length), uIn=U, spongeFraction=0.15, spongeTau=1.0,
                   absorb=0.02, smagorinsky=case.get("smagorinsky", 0.0), forceEvery=case.get("force_every", 1))
        return cfg, sdfs, None if k == "adjoint3d" else _macro3(case, rng), length
    if k == "tunnel2d":
        w, h = case["width"], case["height"]
        cfg = dict(_config2(case), width=w, height=h, precision=case["precision"], smagorinsky=case["smagorinsky"],
                   forceEvery=case["force_every"])
        sdf = np.full(w * h, 1e6, dtype=np.float32)
        if case["mode"] != "cavity":
            y, x = np.mgrid[0:h, 0:w].astype(np.float64)
            off = rng.uniform(-0.5, 0.5, 2)
            sdf = (np.hypot(x - (w / 5 + off[0]), y - (h / 2 + 0.5 + off[1])) - h / 10).astype(np.float32).reshape(-1)
        return [(cfg, sdf, _macro2(w, h, U if case["mode"] == "tunnel" else 0.0, rng))]
    out = []
    for w, h, chord, angle, re in _sizes2(case):
        cfg = dict(width=w, height=h, left=2, right=2, bottom=2, top=2, tau=_tau(re, U, chord), smagorinsky=case["smagorinsky"],
                   uIn=U, spongeFraction=0.15, spongeTau=1.0, absorb=0.02, forceEvery=case["force_every"])
        out.append((cfg, _section2(w, h, chord, angle, rng.uniform(-0.5, 0.5, 2)), _macro2(w, h, U, rng)))
    return out


def _pinned(a):
    p = pinned_empty(a.size, a.dtype)
    p[:] = a
    return p


def prepare(case, seed):
    k = case["kind"]
    if k in ("tunnel3d", "moving3d", "adjoint3d"):
        cfg, sdfs, macro, length = _inputs(case, seed)
        s = Solver3D.create(case["width"], case["height"], case["depth"], **cfg)
        st = {"case": case, "solver": s, "sdfs": [_pinned(a) for a in sdfs], "passes": 0}
        if k != "adjoint3d":
            s.setSdf(sdfs[0])
            s.initField(macro)
            st["macro"] = pinned_empty(4 * s.N, np.float32)
        else:
            st["scale"] = 2 / (U * U * math.pi * (length / 2) ** 2)
        s.synchronize()
        return st
    inputs = _inputs(case, seed)
    if k == "tunnel2d":
        cfg, sdf, macro = inputs[0]
        s = Solver.create(**cfg)
        s.setSdf(sdf)
        s.initField(macro)
        s.synchronize()
        return {"case": case, "solver": s, "macro": pinned_empty(4 * s.N, np.float32)}
    b = Batch2D([cfg for cfg, _, _ in inputs])
    for t, (_, sdf, macro) in zip(b.tunnels, inputs):
        t.setSdf(sdf)
        t.initField(macro)
    b.synchronize()
    ends = np.cumsum([0] + [4 * t.N for t in b.tunnels])
    field = pinned_empty(int(ends[-1]), np.float32)
    return {"case": case, "batch": b, "macro": field, "parts": [field[ends[i]:ends[i + 1]] for i in range(len(b.tunnels))]}


# ------------------------------------------------------------------------------------------- the pass


def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "adjoint3d":
        s = state["solver"]
        s.setSdf(state["sdfs"][0])
        s.initField()
        n = case["steps"]
        j = s.adjointForward(n, n - case["window"] + 1, n, checkpointEvery=case["every"], scale=state["scale"])
        g = s.adjointBackward()
        return {"J": j, "dsdf": g["dsdf"].astype(np.float32), "du": g["du"]}
    if k == "batch2d":
        b = state["batch"]
        b.run(case["steps"])
        for t, part in zip(b.tunnels, state["parts"]):
            t.readMacro(part)
        out = {"macro": state["macro"]}
        if case["force_every"]:
            f = np.concatenate([t.readForcesArray() for t in b.tunnels])
            out["steps"], out["force"] = f[:, 0].astype(np.int64), f[:, 1:].astype(np.float32)
        return out
    s = state["solver"]
    if k == "moving3d":
        s.setSdf(state["sdfs"][1 + state["passes"] % 2])
        state["passes"] += 1
    s.run(case["steps"])
    out = {}
    if case["force_every"]:
        f = s.readForcesArray()
        out["steps"] = f[:, 0].astype(np.int64)
        out["force"] = f[:, 1:].astype(np.float64 if case["precision"] == "fp64" else np.float32)
    out["macro"] = s.readMacro(state["macro"])
    return out


def work(case):
    """Bytes: the populations once in and once out, the SDF where the pass sets it, the field and the
    samples that it returns; operations: the collision of every cell update (about 230 for 19
    directions, 110 for 9; the subgrid model about 70 and 40 more). A gradient steps every state
    twice (run and recompute) and sweeps back over it once, at about twice a step's operations."""
    k = case["kind"]
    if k in ("tunnel3d", "moving3d", "adjoint3d"):
        n = case["width"] * case["height"] * case["depth"]
        pops = 19 * {"fp32": 4, "fp16": 2, "bf16": 2, "fp64": 8}[case["precision"]] * n
        flops = (230 + (70 if case.get("smagorinsky") else 0)) * n * case["steps"]
        if k == "adjoint3d":
            return {"bytes": 4 * n + 2 * pops * (case["steps"] // case["every"]) + 8 * n, "flops": 4 * flops}
        return {"bytes": 2 * pops + 16 * n + (4 * n if k == "moving3d" else 0), "flops": flops}
    cells = case["width"] * case["height"] if k == "tunnel2d" else sum(w * h for w, h, *_ in _sizes2(case))
    size = 8 if case.get("precision") == "fp64" else 4
    return {"bytes": 2 * 9 * size * cells + 16 * cells, "flops": (110 + (40 if case["smagorinsky"] else 0)) * cells * case["steps"]}


# -------------------------------------------------------------------------------- 64-bit evaluation

C3 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0), (1, 0, 1),
      (-1, 0, -1), (0, 1, 1), (0, -1, -1), (1, -1, 0), (-1, 1, 0), (1, 0, -1), (-1, 0, 1), (0, 1, -1), (0, -1, 1)]
C2 = [(0, 0), (1, 0), (0, 1), (-1, 0), (0, -1), (1, 1), (-1, 1), (-1, -1), (1, -1)]
W3 = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
W2 = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4
PAIRS3 = [(i, i + 1) for i in range(1, 19, 2)]
PAIRS2 = [(1, 3), (2, 4), (5, 7), (6, 8)]


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _smooth(t):
    t = t.clamp(0, 1)
    return t * t * (3 - 2 * t)


class _Flow:
    """Link tables and the step of a set of cells (one 3D box, or the 2D boxes of a batch laid end to
    end) in float64. ``src`` holds, per direction and cell, the element that the cell pulls; the links
    across a body wall are interpolated between two elements."""

    def __init__(self, dim):
        self.dim, self.dev = dim, _dev()
        self.c = C3 if dim == 3 else C2
        self.w = W3 if dim == 3 else W2
        self.pairs = PAIRS3 if dim == 3 else PAIRS2
        self.q = len(self.c)
        self.opp = [0] * self.q
        for a, b in self.pairs:
            self.opp[a], self.opp[b] = b, a

    def mirror(self, i, axis):
        v = list(self.c[i])
        v[axis] = -v[axis]
        return self.c.index(tuple(v))

    def feq(self, rho, u):
        usq = 1.5 * sum(v * v for v in u)
        out = []
        for i in range(self.q):
            cu = 3 * sum(a * v for a, v in zip(self.c[i], u))
            out.append(self.w[i] * (rho - 1 + rho * (cu + 0.5 * cu * cu - usq)))
        return torch.stack([o if torch.is_tensor(o) else torch.as_tensor(o) for o in out])

    def link(self, n, rows):
        """rows: per direction, the body links (cell, solid source, next fluid cell or -1, first cell)."""
        cat = lambda k: torch.cat([r[k] for r in rows]) if rows else torch.empty(0, dtype=torch.int64, device=self.dev)  # noqa: E731
        self.lc, self.ls, self.ln = cat(0), cat(1), cat(2)
        li = torch.cat([torch.full_like(r[0], i) for i, r in enumerate(rows, 1)])
        lj = torch.tensor(self.opp, device=self.dev)[li]
        self.lat, self.lj = li * n + self.lc, lj * n + self.lc
        self.li_self = li * n + self.lc
        self.lnext = torch.where(self.ln >= 0, lj * n + self.ln.clamp(min=0), self.lj)
        self.cdir = torch.tensor(self.c, dtype=torch.float64, device=self.dev)[lj]

    def wall(self, sdf):
        df, ds = sdf[self.lc], sdf[self.ls]
        q = (df / (df - ds).clamp(min=1e-6)).clamp(1e-3, 1.0)
        near = q < 0.5
        # q < 1/2: 2q f_j + (1 - 2q) f_j(next), plain bounce-back without a next fluid cell; else from f_i here
        c1 = torch.where(near, torch.where(self.ln >= 0, 2 * q, torch.ones_like(q)), 1 / (2 * q))
        c2 = torch.where(near, torch.where(self.ln >= 0, 1 - 2 * q, torch.zeros_like(q)), (2 * q - 1) / (2 * q))
        return c1, c2, torch.where(near, self.lnext, self.li_self)

    def pull(self, f, wall):
        """The pulled populations and the force on the body of one step from f (q, n)."""
        flat = f.reshape(-1)
        g = flat[self.src]
        c1, c2, e2 = wall
        fj = flat[self.lj]
        fi = c1 * fj + c2 * flat[e2]
        g = g.reshape(-1).index_put((self.lat,), fi).reshape(self.q, -1)
        return g, self.cdir * (fj + fi)[:, None]


class _Flow3(_Flow):
    def __init__(self, w, h, d, cfg, sdf):
        super().__init__(3)
        self.n, self.shape, self.cfg = w * h * d, (w, h, d), cfg
        idx = torch.arange(self.n, device=self.dev)
        self.x, self.y, self.z = idx % w, idx // w % h, idx // (w * h)
        self.tau, self.cs2 = cfg["tau"], cfg["smagorinsky"] ** 2
        self.lam = min(3 / 16, 50 * (self.tau - 0.5) ** 2)
        start = (w - 1) * (1 - cfg["spongeFraction"])
        s = _smooth((self.x.double() - start) / (w - 1 - start))
        self.om = 1 / (self.tau * (1 - s) + cfg["spongeTau"] * s)
        self.sigma = cfg["absorb"] * s * s
        self.inlet, self.outlet = self.x == 0, self.x == w - 1
        self.geometry(sdf)

    def geometry(self, sdf):
        w, h, d = self.shape
        n, x, y, z = self.n, self.x, self.y, self.z
        idx = torch.arange(n, device=self.dev)
        solid = (sdf < 0) & ~self.inlet & ~self.outlet
        self.solid = solid
        src = torch.empty((19, n), dtype=torch.int64, device=self.dev)
        src[0] = idx
        rows, self.slip = [], []
        for i in range(1, 19):
            c = C3[i]
            j = self.opp[i]
            sx, sy, sz = x - c[0], y - c[1], z - c[2]
            ox, oy, oz = (sx < 0) | (sx >= w), (sy < 0) | (sy >= h), (sz < 0) | (sz >= d)
            inside = ~(ox | oy | oz)
            s = (sx + w * (sy + h * sz)).clamp(0, n - 1)
            e = torch.where(inside, i * n + s, j * n + idx)
            face = (oy ^ oz) & ~ox
            r = torch.where(oy, sx + w * (y + h * sz), sx + w * (sy + h * z)).clamp(0, n - 1)
            m = torch.where(oy, torch.full_like(r, self.mirror(i, 1)), torch.full_like(r, self.mirror(i, 2)))
            e = torch.where(face & ~solid[r], m * n + r, e)
            out = ox & self.outlet
            e = torch.where(out, i * n + (w - 2) + w * (y + h * z), e)
            src[i] = e
            live = ~solid & ~self.inlet
            at = torch.nonzero(face & solid[r] & live).reshape(-1)
            self.slip.append((j * n + at, C3[j]))
            at = torch.nonzero(inside & solid[s] & live).reshape(-1)
            nx, ny, nz = x[at] + c[0], y[at] + c[1], z[at] + c[2]
            ok = (nx >= 0) & (nx < w) & (ny >= 0) & (ny < h) & (nz >= 0) & (nz < d)
            nn = torch.where(ok, nx + w * (ny + h * nz), torch.zeros_like(nx))
            rows.append((at, s[at], torch.where(ok & ~solid[nn], nn, torch.full_like(nn, -1))))
        self.src = src
        self.link(n, rows)

    def step(self, f, wall, u_in):
        """One step: the new populations and the force (3,)."""
        g, terms = self.pull(f, wall)
        force = terms.sum(0)
        flat = f.reshape(-1)
        for at, c in self.slip:
            if at.numel():
                force = force + torch.tensor(c, dtype=torch.float64, device=self.dev) * (2 * flat[at]).sum()
        drho = g.sum(0)
        rho = 1 + drho
        u = [sum(self.c[i][a] * g[i] for i in range(19) if self.c[i][a]) / rho for a in range(3)]
        usq = 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
        om = self.om
        cu = {a: 3 * sum(k * v for k, v in zip(self.c[a], u) if k) for a, _ in self.pairs}
        eqs = {a: self.w[a] * (drho + rho * (0.5 * cu[a] * cu[a] - usq)) for a in cu}
        eqa = {a: self.w[a] * rho * cu[a] for a in cu}
        if self.cs2 > 0:
            ne = {a: g[a] + g[b] - 2 * eqs[a] for a, b in self.pairs}
            p = lambda k, l: sum(self.c[a][k] * self.c[a][l] * ne[a] for a in ne if self.c[a][k] * self.c[a][l])  # noqa: E731
            pi = torch.sqrt(p(0, 0) ** 2 + p(1, 1) ** 2 + p(2, 2) ** 2 + 2 * (p(0, 1) ** 2 + p(0, 2) ** 2 + p(1, 2) ** 2))
            t0 = 1 / om
            om = 2 / (t0 + torch.sqrt(t0 * t0 + 18 * math.sqrt(2) * self.cs2 * pi / rho))
        omm = 1 / (0.5 + self.lam / (1 / om - 0.5))
        dq = 1.5 * rho * (u_in * u_in) - rho * usq
        new = [g[0] - om * (g[0] - self.w[0] * (drho - rho * usq)) - self.sigma * self.w[0] * dq] + [None] * 18
        eq1 = [-self.w[0] * usq] + [None] * 18
        ui = [self.w[i] * (3 * self.c[i][0] * u_in + (4.5 * self.c[i][0] ** 2 - 1.5) * u_in * u_in) for i in range(19)]
        for a, b in self.pairs:
            sym, asym = om * (0.5 * (g[a] + g[b]) - eqs[a]), omm * (0.5 * (g[a] - g[b]) - eqa[a])
            cut = 3 * self.c[a][0] * u_in
            ss = self.sigma * self.w[a] * (0.5 * rho * (cut * cut - cu[a] * cu[a]) - dq)
            sa = self.sigma * self.w[a] * rho * (cut - cu[a])
            new[a], new[b] = g[a] - sym - asym + ss + sa, g[b] - sym + asym + ss - sa
            t = 0.5 * cu[a] * cu[a] - usq
            eq1[a], eq1[b] = self.w[a] * (t + cu[a]), self.w[b] * (t - cu[a])
        out = []
        for i in range(19):
            v = torch.where(self.outlet, eq1[i], new[i])
            v = torch.where(self.inlet, ui[i] * torch.ones_like(v), v)
            out.append(torch.where(self.solid, f[i], v))
        return torch.stack(out), force

    def macro(self, f):
        rho = 1 + f.sum(0)
        m = torch.stack([sum(self.c[i][a] * f[i] for i in range(19)) / rho for a in range(3)] + [rho], 1)
        return torch.where(self.solid[:, None], torch.zeros_like(m), m)

    def start(self, macro):
        m = torch.as_tensor(macro, device=self.dev).double().reshape(-1, 4).T
        return torch.where(self.solid, torch.zeros(1, dtype=torch.float64, device=self.dev), self.feq(m[3], m[:3]))

    def move(self, f, sdf):
        """A new obstacle: cells that it uncovers start from the mean of their fluid neighbours."""
        m, old = self.macro(f), self.solid
        w, h, d = self.shape
        self.geometry(sdf)
        at = torch.nonzero(old & ~self.solid).reshape(-1)
        total = torch.zeros((at.numel(), 5), dtype=torch.float64, device=self.dev)
        for c in C3[1:]:
            x, y, z = self.x[at] + c[0], self.y[at] + c[1], self.z[at] + c[2]
            ok = (x >= 0) & (x < w) & (y >= 0) & (y < h) & (z >= 0) & (z < d)
            v = m[torch.where(ok, x + w * (y + h * z), torch.zeros_like(x))]
            ok = ok & (v[:, 3] != 0)
            total += torch.cat([v, torch.ones_like(v[:, :1])], 1) * ok[:, None]
        some = total[:, 4] > 0
        mean = total[:, :4] / total[:, 4:].clamp(min=1)
        rho = torch.where(some, mean[:, 3], torch.ones_like(mean[:, 3]))
        u = [torch.where(some, mean[:, a], torch.full_like(rho, U if a == 0 else 0.0)) for a in range(3)]
        f = f.clone()
        f[:, at] = self.feq(rho, u)
        return f


class _Flow2(_Flow):
    def __init__(self, inputs):
        super().__init__(2)
        base, parts = 0, []
        for cfg, sdf, macro in inputs:
            parts.append(self.box(cfg, torch.as_tensor(sdf, device=self.dev).double(), base))
            base += cfg["width"] * cfg["height"]
        self.n = base
        cat = lambda k: torch.cat([p[k] for p in parts])  # noqa: E731
        self.om, self.sigma, self.target, self.inlet, self.outlet, self.solid = (cat(k) for k in ("om", "sigma", "target", "inlet", "outlet", "solid"))
        self.lam = cat("lam")
        self.cs2, self.force = inputs[0][0].get("smagorinsky", 0.0) ** 2, inputs[0][0].get("bodyForce", (0.0, 0.0))
        # box() numbers elements (direction, cell); the flat element is direction * n + cell
        self.src = torch.stack([torch.cat([p["dir"][i] * base + p["cell"][i] for p in parts]) for i in range(9)])
        self.add = torch.stack([torch.cat([p["add"][i] for p in parts]) for i in range(9)])
        self.link(base, [tuple(torch.cat([p["rows"][i][k] for p in parts]) for k in range(3)) for i in range(8)])
        self.sdf = cat("sdf")
        self.box_of = torch.cat([torch.full((p["om"].numel(),), k, device=self.dev) for k, p in enumerate(parts)])
        self.boxes = len(parts)
        self.f0 = self.feq(*(lambda m: (m[0], m[1:3]))(torch.cat([torch.as_tensor(m, device=self.dev).double().reshape(-1, 4) for _, _, m in inputs]).T))

    def box(self, cfg, sdf, base):
        w, h = cfg["width"], cfg["height"]
        n = w * h
        idx = torch.arange(n, device=self.dev)
        x, y = idx % w, idx // w
        left, right, bottom, top = cfg["left"], cfg["right"], cfg["bottom"], cfg["top"]
        inlet, outlet = (x == 0) & (left == 2), (x == w - 1) & (right == 2)
        solid = (sdf < 0) & ~inlet & ~outlet
        p = {"solid": solid, "inlet": inlet, "outlet": outlet, "sdf": sdf, "dir": [idx * 0], "cell": [idx + base], "rows": [],
             "add": [torch.zeros(n, dtype=torch.float64, device=self.dev)]}

        def wrap(a, b):
            a = torch.where((a < 0) & (left == 0), a + w, a)
            a = torch.where((a >= w) & (right == 0), a - w, a)
            b = torch.where((b < 0) & (bottom == 0), b + h, b)
            b = torch.where((b >= h) & (top == 0), b - h, b)
            return a, b, (a >= 0) & (a < w) & (b >= 0) & (b < h)

        for i in range(1, 9):
            c, j = C2[i], self.opp[i]
            sx, sy, inside = wrap(x - c[0], y - c[1])
            s = torch.where(inside, sy * w + sx, idx * 0)
            mode = torch.where(sy < 0, torch.full_like(sy, bottom), torch.full_like(sy, top))
            off_y = (sy < 0) | (sy >= h)
            slip, moving = off_y & (mode == 2), off_y & (mode == 3)
            d = torch.where(inside, torch.full_like(idx, i), torch.full_like(idx, j))
            d = torch.where(slip, torch.full_like(idx, self.mirror(i, 1)), d)
            cell = torch.where(inside, s, torch.where(slip, y * w + sx.clamp(0, w - 1), idx))
            p["dir"].append(d)
            p["cell"].append(cell + base)
            p["add"].append(torch.where(moving, 6 * self.w[i] * c[0] * cfg.get("uLid", 0.0), 0.0).double())
            at = torch.nonzero(inside & solid[s] & ~solid).reshape(-1)
            nx, ny, ok = wrap(x[at] + c[0], y[at] + c[1])
            nn = torch.where(ok, ny * w + nx, nx * 0)
            p["rows"].append((at + base, s[at] + base, torch.where(ok & ~solid[nn], nn + base, torch.full_like(nn, -1))))
        tau, start = cfg["tau"], (w - 1) * (1 - cfg.get("spongeFraction", 0.0))
        so = _smooth((x.double() - start) / (w - 1 - start)) if start < w - 1 else torch.zeros(n, dtype=torch.float64, device=self.dev)
        p["om"] = 1 / (tau * (1 - so) + cfg.get("spongeTau", 1.0) * so)
        p["sigma"] = cfg.get("absorb", 0.0) * so * so
        p["target"] = torch.full((n,), float(cfg.get("uIn", 0.0)), dtype=torch.float64, device=self.dev)
        p["lam"] = torch.full((n,), 3 / 16, dtype=torch.float64, device=self.dev)
        return p

    def step(self, f, wall):
        g, terms = self.pull(f, wall)
        g = list((g + self.add).unbind(0))
        u0 = self.target
        r = (1 + g[0] + g[2] + g[4] + 2 * (g[3] + g[6] + g[7])) / (1 - u0)
        v = g[0] + g[2] + g[4] + 2 * (g[1] + g[5] + g[8])
        h = 0.5 * (g[2] - g[4])
        i, o = self.inlet, self.outlet
        g1, g5, g8 = g[3] + 2 / 3 * r * u0, g[7] - h + r * u0 / 6, g[6] + h + r * u0 / 6
        g3, g7, g6 = g[1] - 2 / 3 * v, g[5] + h - v / 6, g[8] - h - v / 6
        for k, a, m in ((1, g1, i), (5, g5, i), (8, g8, i), (3, g3, o), (7, g7, o), (6, g6, o)):
            g[k] = torch.where(m, a, g[k])
        drho = sum(g)
        rho = 1 + drho
        fx, fy = self.force
        ux = (g[1] - g[3] + g[5] - g[6] - g[7] + g[8] + 0.5 * fx) / rho
        uy = (g[2] - g[4] + g[5] + g[6] - g[7] - g[8] + 0.5 * fy) / rho
        usq = 1.5 * (ux * ux + uy * uy)
        om = self.om
        cu = {a: 3 * (C2[a][0] * ux + C2[a][1] * uy) for a, _ in self.pairs}
        eqs = {a: self.w[a] * (drho + rho * (0.5 * cu[a] * cu[a] - usq)) for a in cu}
        if self.cs2 > 0:
            ne = {a: g[a] + g[b] - 2 * eqs[a] for a, b in self.pairs}
            p = lambda k, l: sum(C2[a][k] * C2[a][l] * ne[a] for a in ne)  # noqa: E731
            pi = torch.sqrt(p(0, 0) ** 2 + p(1, 1) ** 2 + 2 * p(0, 1) ** 2)
            t0 = 1 / om
            om = 2 / (t0 + torch.sqrt(t0 * t0 + 18 * math.sqrt(2) * self.cs2 * pi / rho))
        omm = 1 / (0.5 + self.lam / (1 / om - 0.5))
        dq = 1.5 * rho * u0 * u0 - rho * usq
        uf = ux * fx + uy * fy
        new = [g[0] - om * (g[0] - self.w[0] * (drho - rho * usq)) - self.sigma * self.w[0] * dq
               - 3 * (1 - 0.5 * om) * self.w[0] * uf] + [None] * 8
        for a, b in self.pairs:
            cut, cf = 3 * C2[a][0] * u0, C2[a][0] * fx + C2[a][1] * fy
            ss = self.sigma * self.w[a] * (0.5 * rho * (cut * cut - cu[a] * cu[a]) - dq)
            ss = ss + (1 - 0.5 * om) * self.w[a] * (3 * cu[a] * cf - 3 * uf)
            sa = self.sigma * self.w[a] * rho * (cut - cu[a]) + (1 - 0.5 * omm) * self.w[a] * 3 * cf
            sym, asym = om * (0.5 * (g[a] + g[b]) - eqs[a]), omm * (0.5 * (g[a] - g[b]) - self.w[a] * rho * cu[a])
            new[a], new[b] = g[a] - sym - asym + ss + sa, g[b] - sym + asym + ss - sa
        return torch.where(self.solid, f, torch.stack(new)), terms

    def macro(self, f):
        rho = 1 + f.sum(0)
        jx = f[1] - f[3] + f[5] - f[6] - f[7] + f[8] - 0.5 * self.force[0]
        jy = f[2] - f[4] + f[5] + f[6] - f[7] - f[8] - 0.5 * self.force[1]
        m = torch.stack([rho, jx / rho, jy / rho, torch.zeros_like(rho)], 1)
        return torch.where(self.solid[:, None], torch.tensor([1.0, 0, 0, 1.0], dtype=torch.float64, device=self.dev), m)


def _exact_adjoint(case, seed):
    cfg, sdfs, _, length = _inputs(case, seed)
    w, h, d = case["width"], case["height"], case["depth"]
    sdf = torch.as_tensor(sdfs[0], device=_dev()).double()
    flow = _Flow3(w, h, d, cfg, sdf)
    scale = 2 / (U * U * math.pi * (length / 2) ** 2)
    n, first = case["steps"], case["steps"] - case["window"]
    share = scale / case["window"]
    one = torch.ones(flow.n, dtype=torch.float64, device=flow.dev)
    f = torch.where(flow.solid, 0 * one, flow.feq(one, [U * one, 0 * one, 0 * one]))
    every, kept, j = 25, [], 0.0
    with torch.no_grad():
        wall = flow.wall(sdf)
        for k in range(n):
            if k % every == 0:
                kept.append(f)
            f, force = flow.step(f, wall, U)
            if k >= first:
                j += share * float(force[0])
    lam, dsdf, du = torch.zeros_like(f), torch.zeros_like(sdf), 0.0
    for seg in range(len(kept) - 1, -1, -1):
        states = [kept.pop()]
        with torch.no_grad():
            for k in range(seg * every, min(n, (seg + 1) * every) - 1):
                states.append(flow.step(states[-1], wall, U)[0])
        for k in range(min(n, (seg + 1) * every) - 1, seg * every - 1, -1):
            g = states.pop().requires_grad_()
            s = sdf.clone().requires_grad_()
            u = torch.tensor(U, dtype=torch.float64, device=flow.dev, requires_grad=True)
            out, force = flow.step(g, flow.wall(s), u)
            total = (lam * out).sum() + (share * force[0] if k >= first else 0.0)
            lam, gs, gu = torch.autograd.grad(total, [g, s, u])
            dsdf += gs
            du += float(gu)
    return {"J": j, "dsdf": dsdf.cpu().numpy(), "du": du}


def exact(case, seed):
    k, steps, every = case["kind"], case["steps"], case.get("force_every", 1)
    if k == "adjoint3d":
        # beyond about a thousand steps of this grid the taped sweep takes too long
        return _exact_adjoint(case, seed) if case["steps"] * case["width"] * case["height"] * case["depth"] < 6e8 else None
    sampled, forces = [], []
    with torch.no_grad():
        if k in ("tunnel2d", "batch2d"):
            flow = _Flow2(_inputs(case, seed))
            f, wall = flow.f0, flow.wall(flow.sdf)
            box = flow.box_of[flow.lc]
            for t in range(1, steps + 1):
                f, terms = flow.step(f, wall)
                if every and t % every == 0:
                    sampled.append(t)
                    forces.append(torch.zeros((flow.boxes, 2), dtype=torch.float64, device=flow.dev).index_add(0, box, terms))
            out = {"macro": flow.macro(f).reshape(-1).cpu().numpy()}
            if every:
                out["steps"] = np.tile(np.array(sampled, dtype=np.int64), flow.boxes)
                out["force"] = torch.stack(forces, 1).reshape(-1, 2).cpu().numpy()
            return out
        cfg, sdfs, macro, _ = _inputs(case, seed)
        sdfs = [torch.as_tensor(a, device=_dev()).double() for a in sdfs]
        flow = _Flow3(case["width"], case["height"], case["depth"], cfg, sdfs[0])
        f = flow.start(macro)
        sdf = sdfs[0]
        if k == "moving3d":
            sdf = sdfs[1]
            f = flow.move(f, sdf)
        wall = flow.wall(sdf)
        for t in range(1, steps + 1):
            f, force = flow.step(f, wall, U)
            if every and t % every == 0:
                sampled.append(t)
                forces.append(force)
        out = {"macro": flow.macro(f).reshape(-1).cpu().numpy()}
        if every:
            out["steps"] = np.array(sampled, dtype=np.int64)
            out["force"] = torch.stack(forces).cpu().numpy()
        return out
