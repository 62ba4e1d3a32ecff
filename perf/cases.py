"""Timed workloads of the foam step, through the package's public entry points.

A pass is what a program does with one foam (or one batch of foams): load the
initial rows into its context, set the clock, search the neighbours, bootstrap
the Adams-Bashforth history, advance a stretch of accepted steps (with the
rejected attempts, neighbour searches and deletions that fall into it), and
take the energy, the volume and the rows of the snapshot back to the host.
Every pass starts from the same rows, so passes are alike.

Foams are synthetic: uniform positions in a box of the given gas fraction,
radii N(1, std) clipped, the shapes of the benchmark's configurations.
"""
import math

import numpy as np
import torch

import cubble_gb300 as cb

DT0 = 1e-4          # the first step's dt
SKIN = 0.3          # Verlet skin (0.3 <r>)
KAPPA, KPAR, TOL = 0.01, 0.1, 1e-5
FP64, MIXED, FF = 0, 1, 2
# per-dimension radius distribution and deletion threshold of the 2D and 3D
# benchmark configurations
RSTD = {2: 0.1, 3: 0.15}
RCLIP = {2: (0.3, 2.0), 3: (0.3, 2.5)}
RMIN = {2: 0.05, 3: 0.1}


def _case(name, dim, n, steps, precision=FP64, calls=1, phi=None, gas=True, flow=False,
          shear=False, walls="", foams=1):
    c = {"dim": dim, "n": n, "steps": steps, "calls": calls, "precision": precision,
         "phi": phi or (0.9 if dim == 2 else 0.8), "gas": gas, "flow": flow, "shear": shear,
         "walls": walls, "foams": foams}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a small 2D sheet driven one integrate() call per step, as the
        # reference's own loop calls it: launches and call latency
        _case("sheet-2d-1k-calls", 2, 1000, 200, calls=200),
        # the 2D configuration of the benchmark (N = 10^4), both forms
        _case("sheet-2d-10k", 2, 10000, 400),
        _case("sheet-2d-10k-mixed", 2, 10000, 400, precision=MIXED),
        # a 2D channel: walls in x and y, the box-region flow
        _case("channel-2d-40k", 2, 40009, 200, flow=True, walls="xy"),
        # a small 3D foam with float-float pair terms
        _case("foam-3d-4k-ff", 3, 4099, 300, precision=FF),
        # an ordinary 3D foam
        _case("foam-3d-30k", 3, 30011, 200),
        # stabilisation: no gas exchange, no path (what init() runs)
        _case("settle-3d-200k", 3, 200003, 120, gas=False),
        # the headline configuration, 3D N = 10^6, in its three forms
        _case("foam-3d-1m", 3, 1000000, 100),
        _case("foam-3d-1m-mixed", 3, 1000000, 100, precision=MIXED),
        _case("foam-3d-1m-ff", 3, 1000000, 60, precision=FF),
        # the large sheared foam between z walls, shortened
        _case("shear-3d-3m-mixed", 3, 3000017, 50, precision=MIXED, shear=True, walls="z"),
        # a parameter sweep: independent 2D foams of 10^3 ... 3 10^4 bubbles
        # advanced as one batch
        _case("sweep-2d-16-mixed", 2, 0, 300, precision=MIXED, foams=16),
    ]


def draw(rng):
    kind = rng.choice(["plain", "plain", "plain", "flow", "settle", "shear", "sweep"])
    precision = rng.choice([FP64, FP64, MIXED, MIXED, FF])
    dim = rng.choice([2, 3])
    if kind == "sweep":
        return _case(None, 2, 0, rng.randrange(100, 300), precision=precision,
                     foams=rng.randrange(4, 17), phi=round(rng.uniform(0.85, 0.95), 3))
    n = int(math.exp(rng.uniform(math.log(1000), math.log(2000000)))) | 1
    steps = max(40, min(300, int(4e7 / n)))
    steps = rng.randrange(max(30, steps // 2), steps + 1)
    calls = steps if n < 20000 and rng.random() < 0.3 else 1
    walls = rng.choice(["", "", "x", "xy" if dim == 2 else "z"])
    if kind == "shear":
        walls = "y" if dim == 2 else "z"
    phi = round(rng.uniform(0.85, 0.95) if dim == 2 else rng.uniform(0.74, 0.85), 3)
    return _case(None, dim, n, steps, precision=precision, calls=calls, phi=phi,
                 gas=kind != "settle", flow=kind == "flow", shear=kind == "shear", walls=walls)


# ------------------------------------------------------------------ inputs
def _foam(dim, n, phi, seed):
    """Rows and box of one synthetic foam."""
    rng = np.random.default_rng(seed)
    r = np.clip(rng.normal(1.0, RSTD[dim], n), *RCLIP[dim])
    unit = 4.0 / 3.0 * math.pi if dim == 3 else math.pi
    side = float(unit * np.sum(r ** dim) / phi) ** (1.0 / dim)
    pos = [rng.uniform(0.0, side, n) for _ in range(dim)]
    area = 4.0 * math.pi * r * r if dim == 3 else 2.0 * math.pi * r
    box = {"dim": dim, "n": n, "phi": phi, "side": side, "ain": float(np.mean(area)),
           "kappa": KAPPA, "mult": (phi * side ** dim / unit) ** (1.0 / dim)}
    return box, pos, r


def _foams(case, seed):
    """The foams of a case: one, or a sweep over N, phi and kappa."""
    if case["foams"] == 1:
        return [_foam(case["dim"], case["n"], case["phi"], seed)]
    rng = np.random.default_rng(seed + 7919)
    out = []
    for f in range(case["foams"]):
        # sizes on a fixed logarithmic ladder, so that every seed is as much work
        n = int(round(1000.0 * 30.0 ** (f / (case["foams"] - 1.0))))
        box, pos, r = _foam(case["dim"], n, float(rng.uniform(0.85, 0.95)), seed + 104729 * (f + 1))
        box["kappa"] = float(10.0 ** rng.uniform(-3.0, -1.0))
        out.append((box, pos, r))
    return out


def _flow_box(box):
    """The flow region: the middle half of the box, moving along x."""
    s = box["side"]
    lo, hi = (0.25 * s,) * 3, (0.75 * s,) * 3
    return lo, hi, (0.05, 0.0, 0.0)


def _config(case, box):
    s, dim = box["side"], box["dim"]
    lo, hi, vel = _flow_box(box)
    return cb.make_config(
        dimensionality=dim, wall=tuple(int(a in case["walls"]) for a in "xyz"),
        lbb=(0.0, 0.0, 0.0), tfr=(s, s, s if dim == 3 else 0.0), wall_drag=0.1,
        min_rad=RMIN[dim], f0_per_mu0=1.0, k_parameter=KPAR, kappa=box["kappa"],
        skin_radius=SKIN, bubble_volume_multiplier=box["mult"],
        average_surface_area_in=box["ain"], error_tolerance=TOL, time_step=DT0,
        use_gas_exchange=int(case["gas"]), increment_path=int(case["gas"]),
        use_flow=int(case["flow"] or case["shear"]),
        shear_speed=0.05 if case["shear"] else 0.0,
        flow_lbb=lo, flow_tfr=hi, flow_vel=vel if case["flow"] else (0.0, 0.0, 0.0),
        capacity=box["n"], precision=case["precision"], use_graph=1)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64 if a.dtype == np.float64 else torch.int32,
                    pin_memory=True).numpy()
    t[:] = a
    return t


# the snapshot's rows
ROWS3 = ("x", "y", "z", "r", "dxdt", "dydt", "dzdt", "drdt", "path")
ROWS2 = ("x", "y", "r", "dxdt", "dydt", "drdt", "path")
RATES = ("dxdt", "dydt", "dzdt", "drdt", "path")


def prepare(case, seed):
    foams = _foams(case, seed)
    configs = [_config(case, box) for box, _, _ in foams]
    if case["foams"] == 1:
        batch, sims = None, [cb.GpuFoam(configs[0])]
    else:
        batch = cb.GpuFoamBatch(configs)
        sims = batch.foams
    rows = ROWS3 if case["dim"] == 3 else ROWS2
    states, outs = [], []
    for box, pos, r in foams:
        st = {"x": _pinned(pos[0]), "y": _pinned(pos[1]), "r": _pinned(r),
              "z": _pinned(pos[2] if case["dim"] == 3 else np.zeros(box["n"]))}
        states.append(st)
        out = {k: _pinned(np.zeros(box["n"])) for k in rows}
        out["index"] = _pinned(np.zeros(box["n"], np.int32))
        if case["precision"] != MIXED:
            out["num_neighbors"] = _pinned(np.zeros(box["n"], np.int32))
        outs.append(out)
    return {"case": case, "batch": batch, "sims": sims, "states": states, "outs": outs}


def run(state):
    case = state["case"]
    for sim, st in zip(state["sims"], state["states"]):
        sim.load_state(st)
        sim.set_time(DT0)
        sim.search_neighbors()
        sim.bootstrap()
    if state["batch"] is not None:
        reports = state["batch"].integrate(case["steps"])
    else:
        for _ in range(case["calls"]):
            reports = [state["sims"][0].integrate(case["steps"] // case["calls"])]
    clock, rows = [], []
    for sim, rep, out in zip(state["sims"], reports, state["outs"]):
        clock.append([rep["time_integer"] + rep["time_fraction"], rep["time_step"],
                      sim.energy(), sim.total_volume()])
        rows.append(sim.get_state(rows=tuple(out), out=out))
    got = {k: np.concatenate([r[k] for r in rows]) if len(rows) > 1 else rows[0][k]
           for k in rows[0]}
    if case["precision"] == MIXED:  # FP32 rates (and path increments) in this form
        got.update({k: got[k].astype(np.float32) for k in RATES if k in got})
    got["clock"] = np.array(clock)
    got["count"] = np.array([rep["count"] for rep in reports], np.int32)
    return got


def work(case):
    """Per accepted step and bubble: the state read and written once (position,
    radius, rates, previous rates, path, error, saved position) and the pair
    list; the rows loaded and taken back once per pass."""
    dim, total = case["dim"], case["n"]
    if case["foams"] > 1:
        total = sum(int(round(1000.0 * 30.0 ** (f / (case["foams"] - 1.0))))
                    for f in range(case["foams"]))
    pairs = 4.67 if dim == 3 else 2.5  # listed pairs per bubble
    per = (224 if dim == 3 else 176) if case["precision"] != MIXED else (176 if dim == 3 else 136)
    once = 8 * (2 * (dim + 1) + (dim + 1) + 1) + 8
    flops = (45 if dim == 3 else 38) * 0.7 * pairs + (70 if dim == 3 else 55)
    return {"bytes": float(total) * (case["steps"] * (per + 8 * pairs) + once),
            "flops": float(total) * case["steps"] * flops}


# ------------------------------------------------------------------- exact
class _Exact:
    """The same stretch in plain torch, 64-bit throughout."""

    def __init__(self, case, box, pos, r):
        self.c, self.dim, self.L = case, box["dim"], box["side"]
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.tensor(a, dtype=torch.float64, device=self.dev)  # noqa: E731
        self.box = box
        self.x = torch.stack([t(p) for p in pos])
        self.r = t(r)
        n = len(r)
        self.v = torch.zeros(self.dim + 1, n, dtype=torch.float64, device=self.dev)
        self.vo = self.v.clone()
        self.path, self.idx = self.r * 0, torch.arange(n, device=self.dev)
        self.dt, self.time = DT0, 0.0
        self.wall = [a in case["walls"] for a in "xyz"[:self.dim]]

    def order(self, p):
        self.x, self.v, self.vo = self.x[:, p], self.v[:, p], self.vo[:, p]
        self.r, self.path, self.idx = self.r[p], self.path[p], self.idx[p]

    def search(self):
        D, L, n = self.dim, self.L, self.r.numel()
        for a in range(D):
            if not self.wall[a]:
                x = self.x[a]
                self.x[a] = x + L * ((x < 0).double() - (x > L).double())
        cd = int(math.floor(L / (2.0 * float(self.r.max()) + SKIN)))
        dims = [cd] * 3 if D == 3 else [cd, cd, 1]
        while dims[0] * dims[1] * dims[2] > 2 * self.box["n"] + 64:
            dims[dims.index(max(dims))] -= 1
        assert min(dims[:D]) >= 3
        k = [((d * self.x[a]) / L).floor().long().clamp(0, d - 1) for a, d in zip(range(D), dims)]
        cell = k[0] + dims[0] * (k[1] + (dims[1] * k[2] if D == 3 else 0))
        p = torch.argsort(cell, stable=True)
        self.order(p)
        cell, k = cell[p], [q[p] for q in k]
        self.sx, self.sr = self.x.clone(), self.r.clone()
        ncell = dims[0] * dims[1] * dims[2]
        start = torch.zeros(ncell + 1, dtype=torch.long, device=self.dev)
        start[1:] = torch.cumsum(torch.bincount(cell, minlength=ncell), 0)
        me = torch.arange(n, device=self.dev)
        I, J = [], []
        for o in range(3 ** D):
            off, q, ok = [o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1], [], torch.ones_like(me, dtype=torch.bool)
            for a in range(D):
                b = k[a] + off[a]
                if self.wall[a]:
                    ok &= (b >= 0) & (b < dims[a])
                    b = b.clamp(0, dims[a] - 1)
                else:
                    b = b % dims[a]
                q.append(b)
            other = q[0] + dims[0] * (q[1] + (dims[1] * q[2] if D == 3 else 0))
            s = torch.maximum(start[other], me + 1)
            m = torch.where(ok, (start[other + 1] - s).clamp(min=0), 0)
            i = torch.repeat_interleave(me, m)
            j = s[i] + torch.arange(i.numel(), device=self.dev) - (torch.cumsum(m, 0) - m)[i]
            d, cut = self.diff(self.x, i, j), self.r[i] + self.r[j] + SKIN
            near = (d * d).sum(0) < cut * cut
            I.append(i[near])
            J.append(j[near])
        self.i, self.j = torch.cat(I), torch.cat(J)
        self.nn = torch.bincount(self.i, minlength=n) + torch.bincount(self.j, minlength=n)

    def diff(self, x, i, j):
        d = x[:, i] - x[:, j]
        for a in range(self.dim):
            if not self.wall[a]:
                d[a] = torch.where(d[a].abs() > 0.5 * self.L, d[a] - torch.copysign(torch.full_like(d[a], self.L), d[a]), d[a])
        return d

    def pairs(self, x, r, gas, flow):
        """Velocity, pairwise gas flux and overlap sums, flow sums, global sums."""
        D, n = self.dim, r.numel()
        add = lambda a, k, w: a.index_add_(0, k, w)  # noqa: E731
        zero = lambda: torch.zeros(n, dtype=torch.float64, device=self.dev)  # noqa: E731
        fl = [zero() for _ in range(D)]
        if flow:
            for a in range(D):
                add(fl[a], self.j, self.v[a][self.i])
        d = self.diff(x, self.i, self.j)
        m = (d * d).sum(0)
        hit = (r[self.i] + r[self.j]) ** 2 >= m
        i, j, d, m = self.i[hit], self.j[hit], d[:, hit], m[hit]
        r1, r2 = r[i], r[j]
        s = 1.0 / m.sqrt() - 1.0 / (r1 + r2)
        f, g, ov, so, sor = [zero() for _ in range(D)], zero(), zero(), 0.0, 0.0
        for a in range(D):
            add(f[a], i, d[a] * s)
            add(f[a], j, -d[a] * s)
        if flow:
            for a in range(D):
                add(fl[a], i, self.v[a][j])
        if gas:
            q1, q2 = r1 * r1, r2 * r2
            chord = (q2 - (q2 - q1 + m) ** 2 / (4.0 * m)).abs()
            inside = (m < q1) | (m < q2)
            if D == 3:
                oa = math.pi * torch.where(inside, torch.minimum(q1, q2), chord)
            else:
                oa = 2.0 * torch.where(inside, torch.minimum(r1, r2), chord.sqrt())
            w = oa * (1.0 / r2 - 1.0 / r1)
            add(g, i, w)
            add(g, j, -w)
            add(ov, i, oa)
            add(ov, j, oa)
            so, sor = 2.0 * float(oa.sum()), float((oa * (1.0 / r1 + 1.0 / r2)).sum())
        return f, g, ov, fl, so, sor

    def bootstrap(self):
        f = self.pairs(self.x, self.r, False, False)[0]
        f = self.pairs(self.x + self.dt * torch.stack(f), self.r, False, False)[0]
        self.vo[:self.dim] = torch.stack(f)
        self.vo[self.dim] = 0.0
        self.path = self.path * 0

    def boundary(self, v, x, r, fl):
        c, D, L = self.c, self.dim, self.L
        if c["flow"]:
            lo, hi, vel = _flow_box(self.box)
            mult = torch.where(self.nn > 0, 1.0 / self.nn.double(), 0.0)
            inside = torch.ones_like(r, dtype=torch.bool)
            for a in range(D):
                inside &= (((x[a] < hi[a]) & (x[a] > lo[a])) | ((lo[a] - x[a]) ** 2 <= r * r)
                           | ((hi[a] - x[a]) ** 2 <= r * r))
            for a in range(D):
                v[a] = v[a] + torch.where(inside, vel[a], mult * fl[a])
        if c["shear"]:
            v[0] = v[0] + 0.05 * (2.0 * x[D - 1] / L - 1.0)
        drag = torch.ones_like(r)
        for a in range(D):
            if not self.wall[a]:
                continue
            d1, d2 = x[a], x[a] - L
            near = torch.where(d1 * d1 < d2 * d2, d1, d2)
            touch = r * r >= near * near
            sign = torch.where(near < 0, -1.0, 1.0)
            push = sign * (1.0 - near.abs() / r)
            for b in range(D):
                if b != a:
                    v[b] = torch.where(touch, v[b] * 0.9, v[b])
            v[a] = torch.where(touch, v[a] + push * drag, v[a])
            drag = torch.where(touch, drag * 0.9, drag)
        return v

    def step(self):
        c, D = self.c, self.dim
        gas = c["gas"]
        while True:
            h, n = 0.5 * self.dt, self.r.numel()
            xp = self.x + h * (3.0 * self.v[:D] - self.vo[:D])
            rp = self.r + h * (3.0 * self.v[D] - self.vo[D]) if gas else self.r
            f, g, ov, fl, so, sor = self.pairs(xp, rp, gas, c["flow"])
            vp = self.boundary(f, xp, rp, fl)
            vp = torch.stack(vp + [g])
            cx = self.x + h * (self.v[:D] + vp[:D])
            err = (xp - cx).abs().amax(0)
            cr = self.r
            if gas:
                area = 4.0 * math.pi * rp * rp if D == 3 else 2.0 * math.pi * rp
                sa, sar = float(area.sum()), float((area / rp).sum())
                mfa, mfb = (sar - sor) / (sa - so), self.box["kappa"] * self.box["ain"] * n / sa
                vp[D] = ((mfa - 1.0 / rp) * mfb * (area - ov) + vp[D]) * KPAR / area
                cr = self.r + h * (self.v[D] + vp[D])
                err = torch.maximum(err, (rp - cr).abs())
            worst = float(err.max())
            too = worst > TOL
            self.dt *= 0.37 if too else (1.269 if worst < 0.45 * TOL and self.dt < 10 else 1.0)
            if not too:
                break
        grown = float(((cx - self.sx).square().sum(0).sqrt() + (cr - self.sr)).max())
        if gas:
            self.path = self.path + (self.x - cx).square().sum(0).sqrt()
        else:
            vp[D] = self.v[D]
        self.vo, self.v, self.x, self.r = self.v, vp, cx, cr
        self.time += self.dt
        if gas:
            gone = cr <= RMIN[D]
            if bool(gone.any()):
                self.remove(gone)
        if grown >= 0.5 * SKIN:
            self.search()

    def remove(self, gone):
        n = gone.numel()
        left = n - int(gone.sum())
        volume = float((self.r[~gone] ** self.dim).sum())
        p = torch.arange(n, device=self.dev)
        holes = p[:left][gone[:left]]
        back = p[left:][~gone[left:]].flip(0)
        p[holes] = back
        to = torch.arange(n, device=self.dev)
        to[back] = holes
        keep = ~(gone[self.i] | gone[self.j])
        self.i, self.j = to[self.i[keep]], to[self.j[keep]]
        p = p[:left]
        self.order(p)
        self.sx, self.sr, self.nn = self.sx[:, p], self.sr[p], self.nn[p]
        self.r = self.r * (self.box["mult"] / volume ** (1.0 / self.dim))

    def finish(self):
        e = (self.r[self.i] + self.r[self.j] - self.diff(self.x, self.i, self.j).square().sum(0).sqrt()).clamp(min=0)
        unit = 4.0 / 3.0 * math.pi if self.dim == 3 else math.pi
        out = {"x": self.x[0], "y": self.x[1], "r": self.r, "dxdt": self.v[0], "dydt": self.v[1],
               "drdt": self.v[self.dim], "path": self.path, "index": self.idx.int()}
        if self.dim == 3:
            out.update({"z": self.x[2], "dzdt": self.v[2]})
        if self.c["precision"] != MIXED:
            out["num_neighbors"] = self.nn.int()
        out = {k: v.cpu().numpy() for k, v in out.items()}
        return out, [self.time, self.dt, float(2.0 * (e * e).sum()), float(unit * (self.r ** self.dim).sum())]


def exact(case, seed):
    outs, clock = [], []
    for box, pos, r in _foams(case, seed):
        sim = _Exact(case, box, pos, r)
        sim.search()
        sim.bootstrap()
        for _ in range(case["steps"]):
            sim.step()
        out, t = sim.finish()
        outs.append(out)
        clock.append(t)
    got = {k: np.concatenate([o[k] for o in outs]) for k in outs[0]}
    got["clock"] = np.array(clock)
    got["count"] = np.array([len(o["r"]) for o in outs], np.int32)
    return got
