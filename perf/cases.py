"""Performance cases of the filament path: what a user's program has it do.

Each case is a dict of plain values.  prepare() makes what such a program holds
before the call (points, links, a context or a filament system), run() is one
pass through the public entry points, and exact() gives the same outputs in 64
bits from plain torch.  Sizes are those of the benchmark configurations
(qvort_b200/workloads.py) and of ranges around them.

kind        the program it stands for
steps       a driver advancing one small system between two outputs
velocity    a torch program evaluating the filament velocity on the device
adjoint     the same with its gradient (one velocity and its vector-Jacobian product)
gradient    the gradient of a trajectory's loss (adjoint.gradient), drawn only
step        a host driver that keeps f(:) itself: the next step of the default loop with
            its reconnections, state up and down through qv_step_exchange
field       velocity and exact Jacobian at quasiparticles
mesh        the velocity on a mesh of points from the tree
batch       an ensemble of independent systems advanced together
"""
from __future__ import annotations

import math

import numpy as np
import torch

from qvort_b200 import adjoint as A
from qvort_b200 import lib as L
from qvort_b200 import workloads as W

BOX = 0.1


# ------------------------------------------------------------------- the cases
def listed():
    return [
        # The smallest run: one ring of 200 points, open, FP64 (the library's default
        # precision), 20 steps between two outputs.  Launches and latency count.
        dict(name="ring_steps", kind="steps", n=200, pair=False, velocity="BS", precision="fp64",
             order=2, nsteps=20),
        # A small system's velocity: a leap-frogging pair, direct sum, FP64, one call.
        dict(name="pair_velocity", kind="velocity", geometry="pair", n=1000, velocity="BS",
             boundary="open", theta=0.0, precision="fp64", order=2),
        # The tangle (24.7k points, periodic): FP64 Barnes-Hut velocity, the reference's
        # arithmetic and algorithm.
        dict(name="tangle_velocity", kind="velocity", geometry="tangle", n=100, velocity="Tree",
             boundary="periodic", theta=0.4, precision="fp64", order=2),
        # The tangle without a tree (theta = 0): the direct sum over 27 images, FP64 ...
        dict(name="tangle_direct_fp64", kind="velocity", geometry="tangle", n=100, velocity="BS",
             boundary="periodic", theta=0.0, precision="fp64", order=2),
        # ... and in mixed precision.
        dict(name="tangle_direct_mixed", kind="velocity", geometry="tangle", n=100,
             velocity="BS", boundary="periodic", theta=0.0, precision="mixed", order=2),
        # One step of the default loop with the host's copy of the state: the tangle ...
        dict(name="tangle_step", kind="step", geometry="tangle", n=100, theta=0.4,
             precision="mixed"),
        # ... and the large tangle (0.8M points), the largest system of the configurations.
        dict(name="large_step", kind="step", geometry="large", n=3000, theta=0.5,
             precision="mixed"),
        # Velocity and its vector-Jacobian product: 50,000 points through the tree ...
        dict(name="adjoint_tree", kind="adjoint", n=16, points=3125, velocity="Tree", theta=0.4,
             boundary="periodic", precision="mixed", order=2),
        # ... and 6,400 points through the direct sum (the size and precision of the
        # finite-difference check).
        dict(name="adjoint_direct", kind="adjoint", n=16, points=400, velocity="BS", theta=0.0,
             boundary="periodic", precision="fp64", order=2),
        # Quasiparticles in the tangle: velocity and Jacobian at 100 points.
        dict(name="quasiparticles", kind="field", n=100, m=100, boundary="periodic",
             images=False),
        # mesh_velocity's Tree arm on a 32^3 mesh through the tangle.
        dict(name="mesh_tree", kind="mesh", n=100, side=32, boundary="periodic", theta=0.4),
        # The ensemble: 512 open systems of 100 to 8000 points, 10 steps between two outputs.
        dict(name="ensemble", kind="batch", n=512, nmin=100, nmax=8000, nsteps=10),
    ]


def _log(rng, lo, hi):
    """A whole number spread evenly over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "velocity", "velocity", "step", "step", "adjoint", "gradient",
                       "field", "mesh", "batch"])
    bc = rng.choice(["open", "openxy", "openx", "periodic", "periodic"])
    prec = rng.choice(["fp64", "mixed"])
    order = rng.choice([2, 2, 4])
    theta = round(rng.uniform(0.3, 0.6), 3)
    if kind == "steps":
        return dict(kind=kind, n=2 * _log(rng, 32, 500), pair=rng.random() < 0.5,
                    velocity=rng.choice(["BS", "BS", "LIA"]), precision=prec, order=order,
                    nsteps=rng.randint(5, 40))
    if kind == "velocity":
        if rng.random() < 0.5:
            g = rng.choice(["pair", "tangle"])
            return dict(kind=kind, geometry=g, n=2 * _log(rng, 50, 2000) if g == "pair"
                        else _log(rng, 3, 95), velocity="BS",
                        boundary="open" if g == "pair" else bc, theta=0.0, precision=prec,
                        order=order)
        return dict(kind=kind, geometry=rng.choice(["tangle", "large"]), n=_log(rng, 5, 600),
                    velocity="Tree", boundary=bc, theta=theta, precision=prec, order=order)
    if kind == "step":
        return dict(kind=kind, geometry=rng.choice(["tangle", "large"]),
                    n=_log(rng, 5, 600 if prec == "fp64" else 2500), theta=theta, precision=prec)
    if kind == "adjoint":
        tree = rng.random() < 0.6
        return dict(kind=kind, n=rng.randint(2, 16), points=_log(rng, 60, 3000 if tree else 500),
                    velocity="Tree" if tree else "BS", theta=theta if tree else 0.0, boundary=bc,
                    precision=prec, order=order)
    if kind == "gradient":
        tree = rng.random() < 0.5
        return dict(kind=kind, n=rng.randint(2, 16), points=_log(rng, 60, 1500 if tree else 300),
                    velocity="Tree" if tree else "BS", theta=theta if tree else 0.0, boundary=bc,
                    precision=prec, order=order, nsteps=rng.randint(2, 5),
                    every=rng.randint(1, 4))
    if kind == "field":
        images = rng.random() < 0.3
        return dict(kind=kind, n=_log(rng, 4, 20 if images else 95), m=_log(rng, 1, 1000),
                    boundary=bc, images=images)
    if kind == "mesh":
        return dict(kind=kind, n=_log(rng, 10, 150), side=rng.randint(6, 30), boundary=bc,
                    theta=theta)
    return dict(kind=kind, n=_log(rng, 16, 480), nmin=100, nmax=_log(rng, 1000, 8000),
                nsteps=rng.randint(3, 10))


# ------------------------------------------------------------------ their inputs
def _points(case, seed):
    """The workload (points, links, run parameters) of a case."""
    kind = case["kind"]
    if kind == "steps":
        n = case["n"]
        w = (W.leap_frog(n, 0.01, 2 * np.pi * 0.01 / (n // 2), seed) if case["pair"]
             else W.ring(n, 0.01, 1e-5, seed))
        if case["pair"]:
            w.x += np.random.default_rng(seed).uniform(-1e-6, 1e-6, w.x.shape)
        w.params.update(dt=min(1e-7, 0.5 * W.dt_max(w)))
    elif kind in ("adjoint", "gradient"):
        w = W.trefoil_rings(seed, case["n"], case["points"], smooth=True)  # crosses no face
        w.params.update(dt=min(1e-7, 0.5 * W.dt_max(w)))
    elif case.get("geometry") == "pair":
        n = case["n"]
        w = W.leap_frog(n, 0.01, 2 * np.pi * 0.01 / (n // 2), seed)
        w.x += np.random.default_rng(seed).uniform(-1e-6, 1e-6, w.x.shape)
    else:
        w = _rings(case, seed)
    p = dict(velocity=case.get("velocity", "Tree"), boundary=case.get("boundary", "periodic"),
             tree_theta=case.get("theta", 0.0), precision=case.get("precision", "fp64"),
             deriv_order=case.get("order", 2), box_size=BOX)
    if kind == "steps":
        p["boundary"] = "open"
    if kind == "field":
        p["velocity"] = "BS"
    w.params.update(p)
    return w


def _rings(case, seed):
    """The tangles of the benchmark configurations (W.random_rings) with radii spread evenly
    over their range, so that a case has the same number of points for every seed."""
    rmin, rmax, delta = (0.004, 0.015, 3e-4) if case.get("geometry") == "large" else (
        0.008, 0.02, 5e-4)
    k = case["n"]
    radius = rmin + (np.arange(k) + 0.5) / k * (rmax - rmin)
    m = np.maximum(5, np.rint(2 * np.pi * radius / (0.75 * delta)).astype(int))
    rng = np.random.default_rng(seed)
    # no ring crosses an open face
    side = BOX if case.get("boundary", "periodic") == "periodic" else 0.059
    centre = rng.uniform(-side / 2, side / 2, (k, 3))
    e = np.linalg.qr(rng.normal(size=(k, 3, 2)))[0]
    start = np.cumsum(m) - m
    ring = np.repeat(np.arange(k), m)
    i = np.arange(m.sum()) - start[ring]
    t = np.pi * (2 * i + 1) / m[ring]
    x = centre[ring] + radius[ring, None] * (np.sin(t)[:, None] * e[ring, :, 0]
                                             + np.cos(t)[:, None] * e[ring, :, 1])
    inf = (start[ring] + (i + 1) % m[ring] + 1).astype(np.int32)
    beh = (start[ring] + (i - 1) % m[ring] + 1).astype(np.int32)
    return W.Workload("rings", W.wrap(x, BOX), inf, beh,
                      dict(dt=1e-7, delta=delta, quant_circ=W.GAMMA_HE4, corea=W.CORE_A))


def _pinned(a):
    """A page-locked host copy of an array (what a host driver exchanges with the GPU)."""
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _upstream(w, seed):
    """The gradient that comes back to the velocity."""
    return np.random.default_rng(seed + 1).normal(0.0, 0.1, w.x.shape)


def _quasi(case, seed):
    return np.random.default_rng(seed + 2).uniform(-0.45 * BOX, 0.45 * BOX, (case["m"], 3))


def _mesh(case, seed):
    """Cell centres of a side^3 mesh over the box, shifted by the seed's offset."""
    s = case["side"]
    o = np.random.default_rng(seed + 2).uniform(-0.2, 0.2, 3)
    ax = [(np.arange(s) + 0.5 + o[c]) / s * BOX - BOX / 2 for c in range(3)]
    return np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)


def _ensemble(case, seed):
    """The ensemble of the benchmark configuration (W.batch_systems: rings and leap-frogging
    pairs, direct sum below 2000 points, tree above) with sizes spread evenly over the
    logarithm of their range and each time step inside the bound of its own spacing."""
    rng = np.random.default_rng(seed)
    ws = []
    for s in range(case["n"]):
        f = (s + 0.5) / case["n"]
        n = int(round(case["nmin"] ** (1 - f) * case["nmax"] ** f))
        n += n % 2
        R = rng.uniform(0.005, 0.02)
        if s % 2:
            w = W.ring(n, R, 1e-5, seed=int(rng.integers(1 << 30)))
        else:
            w = W.leap_frog(n, R, 2 * np.pi * R / (n // 2))
            w.x += rng.uniform(-1e-7, 1e-7, w.x.shape)
            w.x[:, 2] -= w.x[:, 2].mean()
        w.params["dt"] = min(float(rng.choice([5e-8, 1e-7, 2e-7])), 0.5 * W.dt_max(w))
        if n >= 2000:
            w.params.update(velocity="Tree", tree_theta=0.4)
        ws.append(w)
    return ws


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ws = _ensemble(case, seed)
        b = L.Batch(L.default_params(box_size=BOX, tree_theta=0.4, boundary="open",
                                     quant_circ=W.GAMMA_HE4, corea=W.CORE_A, precision="mixed",
                                     velocity="Tree"),
                    [(w.x, w.infront, w.behind) for w in ws],
                    [w.params["velocity"] for w in ws], [w.params["dt"] for w in ws])
        return dict(case=case, batch=b)
    w = _points(case, seed)
    p = dict(w.params)
    if kind in ("velocity", "adjoint", "gradient"):
        s = dict(case=case, x0=w.x, system=A.FilamentSystem(L.default_params(**p), w.infront,
                                                            w.behind))
        s["x"] = torch.tensor(w.x, device="cuda")
        s["ubar"] = torch.tensor(_upstream(w, seed), device="cuda")
        return s
    if kind in ("field", "mesh"):
        c = L.Context(L.default_params(**p))
        c.set_points(w.x, w.infront, w.behind)
        return dict(case=case, ctx=c, pts=(_quasi if kind == "field" else _mesh)(case, seed))
    # the host's copy of f(:) with room for inserted points, and no history yet
    if kind == "step":
        p["line_ops"] = 2
    cap = w.n + w.n // 50 + 64
    f = {k: np.zeros((cap, 3)) for k in ("x", "u", "u1", "u2", "u3")}
    f.update({k: np.zeros(cap, np.int32) for k in ("infront", "behind", "closest")})
    f["closestd"] = np.zeros(cap)
    for k, v in (("x", w.x), ("infront", w.infront), ("behind", w.behind)):
        f[k][:w.n] = v
    s = dict(case=case, n=w.n, cap=cap, itime=0, ctx=L.Context(L.default_params(**p)),
             f={k: _pinned(v) for k, v in f.items()})
    if kind == "steps":
        s["start"] = {k: s["f"][k].copy() for k in ("x", "infront", "behind")}
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "velocity":
        with torch.no_grad():
            return A.velocity(state["x"], state["system"])
    if kind == "adjoint":
        x = state["x"].detach().requires_grad_(True)
        u = A.velocity(x, state["system"])
        (g,) = torch.autograd.grad(u, x, state["ubar"])
        return u.detach(), g
    if kind == "gradient":
        return A.gradient(state["x0"], state["system"], case["nsteps"], case["every"])
    if kind == "field":
        return state["ctx"].field_velocity(state["pts"], case["images"])
    if kind == "mesh":
        return state["ctx"].field_velocity_tree(state["pts"])
    if kind == "batch":
        state["batch"].step(case["nsteps"])
        return state["batch"].get_points()
    c, f = state["ctx"], state["f"]
    if kind == "steps":
        c.set_state(state["n"], **state["start"])
        c.steps(1, case["nsteps"])
        c.get_state(state["cap"], **f)
        return {k: v[:state["n"]] for k, v in f.items()}
    # the program's next step: f(:) goes in and comes back in place (the first steps of a
    # tangle reconnect its random crossings, the later ones find few)
    state["itime"] += 1
    state["n"] = c.step_exchange(state["itime"], state["n"], state["cap"], f, f)
    return dict(f, n=state["n"])


# ------------------------------------------------------------------- their work
NIMG = {"open": 1, "openxy": 3, "openx": 9, "periodic": 27}
PAIR, PAIR_VJP, LOCAL = 38, 110, 120  # flops of a segment term, of its gradient, of the local term


def _size(case):
    """Mean point count of a case (of its workload's distribution)."""
    if case["kind"] in ("adjoint", "gradient"):
        return case["n"] * case["points"]
    if case["kind"] == "steps" or case.get("geometry") == "pair":
        return case["n"]
    return case["n"] * (267.0 if case.get("geometry") == "large" else 234.5)


def _tree_evals(n, nimg, theta):
    """Terms a target takes from the tree: opened cells per level grow as 1/theta^3, the
    images' as the boundary's count (fitted to the walk's own counts of the tangles)."""
    return 65.0 * (0.4 / theta) ** 1.6 * math.log2(max(n, 4)) * (1 + 0.02 * nimg)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
        mean = (case["nmax"] - case["nmin"]) / (hi - lo)
        at = min(max(math.log(2000.0), lo), hi)  # direct sum below 2000 points, tree above
        pairs = (math.exp(2 * at) - math.exp(2 * lo)) / 2 / (hi - lo)
        tree = (math.exp(hi) - math.exp(at)) / (hi - lo) * _tree_evals(4000, 1, 0.4)
        return dict(bytes=case["n"] * mean * (case["nsteps"] * 80.0 + 48),
                    flops=case["n"] * case["nsteps"] * ((pairs + tree) * PAIR + mean * LOCAL))
    n, nimg = _size(case), NIMG[case.get("boundary", "open" if kind == "steps" else "periodic")]
    tree = case.get("theta", 0.0) > 0
    terms = _tree_evals(n, nimg, case["theta"]) if tree else n * nimg
    if kind == "steps" and case["velocity"] == "LIA":
        terms = 0
    if kind == "velocity":
        return dict(bytes=n * 56.0, flops=n * (terms * PAIR + LOCAL))
    if kind == "adjoint":
        return dict(bytes=n * 104.0, flops=n * (terms * (PAIR + PAIR_VJP) + 10 * LOCAL))
    if kind == "gradient":
        k = case["nsteps"]  # forward, recomputed forward, backward, and the loss's velocity
        return dict(bytes=n * 48.0, flops=n * (2 * k + 1) * (terms * PAIR + LOCAL)
                    + n * (k + 1) * terms * PAIR_VJP)
    if kind == "steps":
        k = case["nsteps"]  # and the search for each point's closest other: 8 flops a pair
        return dict(bytes=n * 260.0, flops=k * n * (terms * PAIR + n * 8 + LOCAL))
    if kind == "step":
        return dict(bytes=n * 248.0, flops=n * (terms * PAIR + LOCAL + 500))
    if kind == "field":
        grad = nimg if case["images"] else 1
        return dict(bytes=n * 32.0 + case["m"] * 120.0,
                    flops=case["m"] * n * (nimg * PAIR + grad * PAIR_VJP))
    m = case["side"] ** 3
    return dict(bytes=n * 32.0 + m * 48.0, flops=m * terms * PAIR)


# -------------------------------------------------- the same in 64 bits, in torch
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _cross(a, b):
    return torch.stack([a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1],
                        a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2],
                        a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]], -1)


def _shifts(boundary):
    """The boundary's image shifts, the unshifted one first."""
    r = {"open": (0, 0, 0), "openxy": (0, 0, 1), "openx": (0, 1, 1), "periodic": (1, 1, 1)}
    a, b, c = r[boundary]
    s = [(i, j, k) for i in range(-a, a + 1) for j in range(-b, b + 1) for k in range(-c, c + 1)]
    s.sort(key=lambda t: t != (0, 0, 0))
    return torch.tensor(s, dtype=torch.float64, device=_dev()) * BOX


class _System:
    """A case's points, links and ghosts in torch."""

    def __init__(self, w, x=None):
        self.w, self.p = w, w.params
        self.x = torch.tensor(w.x, device=_dev()) if x is None else x
        self.inf = torch.tensor(w.infront, device=_dev()).long() - 1
        self.beh = torch.tensor(w.behind, device=_dev()).long() - 1
        self.sh = _shifts(self.p["boundary"])
        self.gi, self.gb = self._ghost(self.inf), self._ghost(self.beh)
        self.gii = self._ghost(self.inf[self.inf])
        self.gbb = self._ghost(self.beh[self.beh])

    def _ghost(self, at):
        g = self.x[at]
        axes = {"open": 0, "openxy": 1, "openx": 2, "periodic": 3}[self.p["boundary"]]
        for c in range(3 - axes, 3):
            d = (self.x[:, c] - g[:, c]).detach()
            shift = (d > BOX / 2).double() * BOX - (d < -BOX / 2).double() * BOX
            g = g + torch.nn.functional.one_hot(torch.tensor(c, device=g.device), 3) * shift[:, None]
        return g

    def local(self):
        """The local term: beta s' x s'' on non-uniform finite differences."""
        x, gi, gb = self.x, self.gi, self.gb
        i, b = (x - gi).norm(dim=1, keepdim=True), (x - gb).norm(dim=1, keepdim=True)
        if self.p["deriv_order"] == 2:
            s1 = (b * gi + (i - b) * x - i * gb) / (2 * b * i)
            s2 = 2 * (gi / (i * (i + b)) - x / (i * b) + gb / (b * (i + b)))
        else:
            # Lagrange weights of the five points at -b-bb, -b, 0, i, i+ii
            ii = (self.gii - gi).norm(dim=1, keepdim=True)
            bb = (self.gbb - gb).norm(dim=1, keepdim=True)
            t = [-b - bb, -b, torch.zeros_like(b), i, i + ii]
            f = [self.gbb, gb, x, gi, self.gii]
            w1, w2 = [], []
            for a in range(5):
                o = [t[q] for q in range(5) if q != a]
                den = (t[a] - o[0]) * (t[a] - o[1]) * (t[a] - o[2]) * (t[a] - o[3])
                e3 = o[0] * o[1] * o[2] + o[0] * o[1] * o[3] + o[0] * o[2] * o[3] + o[1] * o[2] * o[3]
                e2 = o[0] * o[1] + o[0] * o[2] + o[0] * o[3] + o[1] * o[2] + o[1] * o[3] + o[2] * o[3]
                w1.append(-e3 / den)
                w2.append(2 * e2 / den)
            w1[2], w2[2] = -sum(w1[:2] + w1[3:]), -sum(w2[:2] + w2[3:])
            s1 = sum(a * q for a, q in zip(w1, f))
            s2 = sum(a * q for a, q in zip(w2, f))
        G, a = self.p["quant_circ"], self.p["corea"]
        if self.p["velocity"] == "LIA":
            beta = G / (4 * math.pi) * torch.log(1 / s2.norm(dim=1, keepdim=True) / a)
        else:
            beta = G / (4 * math.pi) * torch.log(1.21 / a * torch.sqrt(i * b))
        return beta * _cross(s1, s2)


def _segment(r1, r2, s):
    """(|R1|+|R2|) / (|R1||R2| (|R1||R2| + R1.R2)) R1 x s, without cancellation either way."""
    a, b, d = r1.norm(dim=-1), r2.norm(dim=-1), (r1 * r2).sum(-1)
    c = _cross(r1, s)
    ab = a * b
    safe = torch.where(d < 0, ab - d, torch.ones_like(d))
    den = torch.where(d < 0, (c * c).sum(-1) / safe, ab + d)
    ok = den > 0
    f = torch.where(ok, (a + b) / (ab * torch.where(ok, den, torch.ones_like(den))),
                    torch.zeros_like(den))
    return f[..., None] * c


def _direct(sy, lo, hi, k):
    """What image k of the direct sum adds to the velocity of points lo..hi."""
    t = torch.arange(lo, hi, device=sy.x.device)
    j = torch.arange(sy.x.shape[0], device=sy.x.device)
    skip = j[None] == sy.beh[t][:, None]
    if k == 0:
        skip = skip | (j[None] == t[:, None])
    skip = skip[..., None]
    s = (sy.gi - sy.x)[None]
    r1 = (sy.x + sy.sh[k])[None] - sy.x[lo:hi, None]
    r1 = torch.where(skip, torch.ones_like(r1), r1)  # a point with itself: a finite gradient
    u = torch.where(skip, torch.zeros_like(r1), _segment(r1, r1 + s, s.expand_as(r1)))
    return u.sum(1) * (sy.p["quant_circ"] / (4 * math.pi))


def _direct_u(w, x=None, ubar=None):
    """The BS arm's velocity of every point and, given ubar, its vector-Jacobian product."""
    grad = ubar is not None
    x = (_System(w).x if x is None else x).detach().requires_grad_(grad)
    sy = _System(w, x)
    local = sy.local()
    u = local.detach().clone()
    g = torch.autograd.grad(local, x, ubar)[0] if grad else None
    n = x.shape[0]
    step = max(1, (4_000_000 if grad else 12_000_000) // n)
    for lo in range(0, n, step):
        hi = min(n, lo + step)
        for k in range(len(sy.sh)):
            part = _direct(_System(w, x) if grad else sy, lo, hi, k)
            u[lo:hi] += part.detach()
            if grad:
                g += torch.autograd.grad(part, x, ubar[lo:hi])[0]
    return (u, g) if grad else u


class _Tree:
    """The octree's cells and moments, level by level."""

    def __init__(self, sy):
        x, s = sy.x, sy.gi - sy.x
        xd = x.detach()
        n = x.shape[0]
        node = torch.zeros(n, dtype=torch.long, device=x.device)
        pts = torch.arange(n, device=x.device)
        corner = torch.full((1, 3), -BOX / 2, dtype=torch.float64, device=x.device)
        width = BOX
        base = 0
        cols = dict(count=[torch.tensor([n], device=x.device)], corner=[corner],
                    width=[torch.full((1,), BOX, dtype=torch.float64, device=x.device)],
                    first=[torch.zeros(1, dtype=torch.long, device=x.device)],
                    parent=[torch.full((1,), -1, dtype=torch.long, device=x.device)])
        cent = [xd.mean(0, keepdim=True)]
        circ, C = [torch.zeros_like(cent[0])], [torch.zeros(1, 9, dtype=torch.float64, device=x.device)]
        while True:
            keep = cols["count"][-1][node] > 1
            node, pts = node[keep], pts[keep]
            if not len(pts):
                break
            lo = corner[node]
            up = lo + width / 2
            hi = xd[pts] >= up
            inside = (xd[pts] >= torch.where(hi, up, lo)) & (xd[pts] < torch.where(hi, up, lo) + width / 2)
            ok = inside.all(1)
            node, pts, hi = node[ok], pts[ok], hi[ok].long()
            key = node * 8 + hi[:, 0] + 2 * hi[:, 2] + 4 * hi[:, 1]
            ids, child, cnt = torch.unique(key, return_inverse=True, return_counts=True)
            up_ids = ids // 8
            half = width / 2
            bit = torch.stack([ids & 1, (ids >> 2) & 1, (ids >> 1) & 1], 1).double()
            corner = corner[up_ids] + bit * half
            width = half
            m = len(ids)
            z3 = torch.zeros(m, 3, dtype=torch.float64, device=x.device)
            ce = z3.index_add(0, child, x[pts]) / cnt[:, None]
            ci = z3.index_add(0, child, s[pts])
            raw = torch.zeros(m, 9, dtype=torch.float64, device=x.device).index_add(
                0, child, (x[pts][:, :, None] * s[pts][:, None, :]).reshape(-1, 9))
            cent.append(ce)
            circ.append(ci)
            C.append(raw - (ce[:, :, None] * ci[:, None, :]).reshape(-1, 9))
            first = torch.full((m,), n, dtype=torch.long, device=x.device).scatter_reduce(
                0, child, pts, "amin")
            cols["count"].append(cnt)
            cols["corner"].append(corner)
            cols["width"].append(torch.full((m,), width, dtype=torch.float64, device=x.device))
            cols["first"].append(first)
            cols["parent"].append(up_ids + base)
            base += len(cols["count"][-2])
            node = child
        for k, v in cols.items():
            setattr(self, k, torch.cat(v))
        self.cent, self.circ, self.C = torch.cat(cent), torch.cat(circ), torch.cat(C)
        m = len(self.count)
        self.nchild = torch.bincount(self.parent[1:], minlength=m)
        self.child0 = torch.cumsum(self.nchild, 0) - self.nchild + 1
        mid = self.corner + self.width[:, None] / 2
        self.geo = (self.cent.detach() - mid).norm(dim=1)

    def visit(self, at, sh, theta, extra):
        """(targets, cells) of the far and of the leaf terms that points `at` take for shift sh."""
        t = torch.arange(at.shape[0], device=at.device)
        c = torch.zeros_like(t)
        far, leaf = [], []
        cent = self.cent.detach() + sh
        while len(t):
            dist = (at[t] - cent[c]).norm(dim=1)
            if extra:
                r = dist - self.geo[c]
                th = self.width[c] / torch.where(r > 0, r, dist)
                go = torch.ones_like(t, dtype=torch.bool)
            else:
                th = self.width[c] / dist
                go = ~(dist < 2.220446049250313e-16)
            one = self.count[c] == 1
            is_far = ~one & (th < theta) & go
            leaf.append(torch.stack([t[one & go], c[one & go]]))
            f = is_far & (c > 0)
            far.append(torch.stack([t[f], c[f]]))
            op = ~one & ~is_far & go
            t, c = t[op], c[op]
            k = self.nchild[c]
            rep = torch.repeat_interleave(torch.arange(len(c), device=at.device), k)
            off = torch.arange(len(rep), device=at.device) - (torch.cumsum(k, 0) - k)[rep]
            t, c = t[rep], self.child0[c[rep]] + off
        return torch.cat(far, 1), torch.cat(leaf, 1)

    @staticmethod
    def far_term(x, cent, circ, C, sh):
        v = x - (cent + sh)
        r2 = 1 / (v * v).sum(1, keepdim=True)
        r3 = r2 * torch.sqrt(r2)
        M = C.reshape(-1, 3, 3)
        w = torch.stack([M[:, 1, 2] - M[:, 2, 1], M[:, 2, 0] - M[:, 0, 2], M[:, 0, 1] - M[:, 1, 0]], 1)
        z = (v[:, :, None] * M).sum(1)
        return (_cross(circ, v) - w) * r3 + 3 * _cross(v, z) * r3 * r2


def _tree_u(w, ubar=None):
    """The Tree arm's velocity of every point and, given ubar, its vector-Jacobian product
    with the opened cells held."""
    grad = ubar is not None
    x = _System(w).x.requires_grad_(grad)
    sy = _System(w, x)
    tr = _Tree(sy)
    local = sy.local()
    G = sy.p["quant_circ"] / (4 * math.pi)
    # the terms' inputs on their own: their adjoints are summed over images and chunks
    X, GI, ce, ci, C = parts = [t.detach().requires_grad_(grad)
                                for t in (x, sy.gi, tr.cent, tr.circ, tr.C)]
    u = local.detach().clone()

    def add(a, term):
        u.index_add_(0, a, term.detach())
        if grad:
            (term * ubar[a]).sum().backward()

    for sh in sy.sh:
        far, leaf = tr.visit(X.detach(), sh, sy.p["tree_theta"], True)
        for q in torch.split(torch.arange(far.shape[1], device=x.device), 8_000_000):
            a, c = far[0][q], far[1][q]
            add(a, G * tr.far_term(X[a], ce[c], ci[c], C[c], sh))
        a, j = leaf[0], tr.first[leaf[1]]
        ok = (j != a) & (j != sy.beh[a]) & (j != sy.inf[a])
        a, j = a[ok], j[ok]
        s = GI[j] - X[j]
        r1 = X[j] + sh - X[a]
        add(a, G * _segment(r1, r1 + s, s))
    if not grad:
        return u
    ups = [ubar] + [torch.zeros_like(q) if q.grad is None else q.grad for q in parts[1:]]
    (g,) = torch.autograd.grad([local, sy.gi, tr.cent, tr.circ, tr.C], x, ups)
    return u, g + X.grad


def _exact_steps(case, seed):
    """The Adams-Bashforth ladder from zero history, every step from plain torch."""
    w = _points(case, seed)
    x = torch.tensor(w.x, device=_dev())
    dt, hist = w.params["dt"], []
    for _ in range(case["nsteps"]):
        u = _System(w, x).local() if case["velocity"] == "LIA" else _direct_u(w, x)
        h = [u] + hist
        k = len(h) - 1
        if k == 0:
            x = x + dt * u
        elif k == 1:
            x = x + dt * (1.5 * h[0] - 0.5 * h[1])
        elif k == 2:
            x = x + dt * (23 * h[0] - 16 * h[1] + 5 * h[2]) / 12
        else:
            x = x + dt * (55 * h[0] - 59 * h[1] + 37 * h[2] - 9 * h[3]) / 24
        hist = h[:3]
    out = {k: None for k in ("closest", "closestd", "infront", "behind")}
    out.update(x=x.cpu(), u=hist[0].cpu())
    out.update({"u%d" % (k + 1): hist[k].cpu() for k in range(min(3, len(hist)))})
    return out


def _exact_field(case, seed):
    w = _points(case, seed)
    sy = _System(w)
    n = sy.x.shape[0]
    pts = torch.tensor(_quasi(case, seed), device=_dev())
    G = sy.p["quant_circ"] / (4 * math.pi)
    s = (sy.gi - sy.x)[None]
    us, js = [], []
    for lo in range(0, len(pts), max(1, 4_000_000 // n)):
        p = pts[lo:lo + max(1, 4_000_000 // n)].requires_grad_(True)
        u, J = torch.zeros_like(p).detach(), torch.zeros(len(p), 3, 3, dtype=p.dtype, device=p.device)
        for k, sh in enumerate(sy.sh):
            r1 = (sy.x + sh)[None] - p[:, None]
            v = G * _segment(r1, r1 + s, s.expand_as(r1)).sum(1)
            u += v.detach()
            if k == 0 or case["images"]:
                for c in range(3):
                    J[:, c] += torch.autograd.grad(v[:, c].sum(), p, retain_graph=c < 2)[0]
        us.append(u)
        js.append(J)
    return torch.cat(us).cpu(), torch.cat(js).cpu()


def _exact_mesh(case, seed):
    sy = _System(_points(case, seed))
    tr = _Tree(sy)
    pts = torch.tensor(_mesh(case, seed), device=_dev())
    u = torch.zeros_like(pts)
    for sh in sy.sh:
        far, leaf = tr.visit(pts, sh, case["theta"], False)
        for q in torch.split(torch.arange(far.shape[1], device=pts.device), 8_000_000):
            a, c = far[0][q], far[1][q]
            u.index_add_(0, a, tr.far_term(pts[a], tr.cent[c], tr.circ[c], tr.C[c], sh))
        a, j = leaf[0], tr.first[leaf[1]]
        s = sy.gi[j] - sy.x[j]
        r1 = sy.x[j] + sh - pts[a]
        u.index_add_(0, a, _segment(r1, r1 + s, s) / (4 * math.pi))
    return u.cpu(), None


def exact(case, seed):
    kind = case["kind"]
    if kind == "steps":
        return _exact_steps(case, seed)
    if kind == "field":
        return _exact_field(case, seed)
    if kind == "mesh":
        return _exact_mesh(case, seed)
    arm = _tree_u if case.get("velocity") == "Tree" else _direct_u
    if kind == "velocity":
        return arm(_points(case, seed)).cpu()
    if kind == "adjoint":
        w = _points(case, seed)
        u, g = arm(w, ubar=torch.tensor(_upstream(w, seed), device=_dev()))
        return u.cpu(), g.cpu()
    # whole steps with reconnections, trajectories' gradients and the ensemble's steps
    # have no short statement in plain torch
    return None
