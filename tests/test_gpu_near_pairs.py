"""GPU tests of the FP64 derivatives where one pair carries nearly all of a sum: a
target close to either end of a segment (filaments about to reconnect, a
quasiparticle beside a line).

The comparison takes every derivative by a complex step of 1e-40 in 80-bit long
doubles, exact to their 5e-20, from the segment factor written with R1 and R2
themselves.  All coordinates are multiples of 2^-40, so x_j - x_i, ghost_j - x_i and
ghost_j - x_j hold exactly in FP64 and every error is the kernel's own.  Bound:
with R1 and R2 at hand no step of the closed derivatives cancels; a component is a
sum of four products whose factors (a reciprocal root each for |R1| and |R2|, one
division, squares) carry at most about twelve roundings of 1.1e-16, and each
product is at most the largest component, so 48 roundings, 5.4e-15 of the largest.
"""
import numpy as np
import pytest

from qvort_b200 import workloads as W

pytestmark = pytest.mark.gpu

BOX = 0.125
SIDE = 2.0 ** -9  # length of the approached segment, about
TOL = 48 * 2.0 ** -53
CD, LD = np.clongdouble, np.longdouble


def _grid(x):
    return np.round(np.asarray(x) * 2.0 ** 40) / 2.0 ** 40


def _cross(a, b):
    return np.stack([a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1],
                     a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2],
                     a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]], axis=-1)


def _len(a):
    return np.sqrt((a * a).sum(-1))


def _segment(r1, r2):
    """The straight segment's term; the angle's second form where it is obtuse."""
    a, b, d, cr = _len(r1), _len(r2), (r1 * r2).sum(-1), _cross(r1, r2)
    obtuse = d.real < 0
    e = np.where(obtuse, (cr * cr).sum(-1) / np.where(obtuse, a * b - d, 1), a * b + d)
    return ((a + b) / (a * b * e))[..., None] * cr


def _shifts(bc):
    r = {"open": (0, 0, 0), "openxy": (0, 0, 1), "openx": (0, 1, 1), "periodic": (1, 1, 1)}[bc]
    return [np.array([i, j, k], LD) * LD(BOX) for i in range(-r[0], r[0] + 1)
            for j in range(-r[1], r[1] + 1) for k in range(-r[2], r[2] + 1)]


def _system(end, gap, seed):
    """A triangle with a side AB of about SIDE, a target `gap` sides off its end
    (1: A, 2: B) with R1.R2 > |s|^2 / 16, and the target's own far-off filament."""
    rng = np.random.default_rng([end, int(1000 * gap), seed])
    s = rng.normal(size=3)
    s *= SIDE / np.linalg.norm(s)
    A = np.array([0.011, -0.007, 0.004]) + rng.uniform(-1e-3, 1e-3, 3)
    while True:
        v = rng.normal(size=3)
        v *= gap * SIDE / np.linalg.norm(v)
        r1, r2 = (-v, s - v) if end == 1 else (-s - v, -v)
        if r1 @ r2 > 0.065 * SIDE ** 2:
            break
    P = A + v if end == 1 else A + s + v
    x = _grid([A, A + s, A + [0.02, -0.013, 0.017], P, P + [-0.02, 0.015, 0.01],
               P + [-0.03, -0.01, 0.02], P + [-0.02, -0.03, -0.01], P + [0.01, -0.02, -0.03]])
    inf = np.array([2, 3, 1, 5, 6, 7, 8, 4], np.int32)
    beh = np.array([3, 1, 2, 8, 4, 5, 6, 7], np.int32)
    prm = dict(boundary="open", velocity="BS", tree_theta=0.0, box_size=BOX, deriv_order=2,
               quant_circ=W.GAMMA_HE4, corea=W.CORE_A, precision="fp64")
    return W.Workload("near", x, inf, beh, prm), P


def _sum_vjp(w, ubar, bc):
    """d (ubar . u) / dx of the local term and the direct sum (no link crosses the box)."""
    n, f, b = w.n, w.infront - 1, w.behind - 1
    G = LD(w.params["quant_circ"]) / (4 * LD(np.pi))
    core = LD(w.params["corea"])
    own, back = np.eye(n, dtype=bool), np.arange(n)[None] == b[:, None]

    def loss(x):
        gi, gb = x[f], x[b]
        i, h = _len(x - gi)[:, None], _len(x - gb)[:, None]
        s1 = (h * gi + (i - h) * x - i * gb) / (2 * h * i)
        s2 = 2 * (gi / (i * (i + h)) - x / (i * h) + gb / (h * (i + h)))
        u = G * np.log(LD(1.21) / core * np.sqrt(i * h)) * _cross(s1, s2)
        for sh in _shifts(bc):
            skip = (back | own if not sh.any() else back)[..., None]
            r1 = (x + sh)[None] - x[:, None]
            r2 = (gi + sh)[None] - x[:, None]
            r1, r2 = np.where(skip, [LD(1), 0, 0], r1), np.where(skip, [0, LD(1), 0], r2)
            u = u + G * np.where(skip, 0, _segment(r1, r2)).sum(1)
        return (u * ubar).sum()

    g = np.empty((n, 3))
    for k in range(3 * n):
        x = w.x.astype(CD)
        x.flat[k] += CD(1e-40j)
        g.flat[k] = float(loss(x).imag / LD(1e-40))
    return g


@pytest.mark.parametrize("bc", ["open", "openxy", "openx", "periodic"])
@pytest.mark.parametrize("gap", [0.07, 0.2, 0.5])
@pytest.mark.parametrize("end", [1, 2])
def test_gradient_of_a_pair_near_a_segments_end(end, gap, bc):
    import torch

    from qvort_b200 import adjoint as A
    from qvort_b200 import lib as L

    for seed in range(4):
        w, _ = _system(end, gap, seed)
        w.params["boundary"] = bc
        ubar = _grid(np.random.default_rng(seed).uniform(-1, 1, w.x.shape))
        s = A.FilamentSystem(L.default_params(**w.params), w.infront, w.behind)
        x = torch.tensor(w.x, device="cuda", requires_grad=True)
        (g,) = torch.autograd.grad(A.velocity(x, s), x, torch.tensor(ubar, device="cuda"))
        s.close()
        og = _sum_vjp(w, ubar, bc)
        assert np.abs(g.cpu().numpy() - og).max() <= TOL * np.abs(og).max()


@pytest.mark.parametrize("theta", [0.3, 0.6])
@pytest.mark.parametrize("gap", [0.07, 0.2, 0.5])
@pytest.mark.parametrize("end", [1, 2])
def test_tree_gradient_of_a_pair_near_a_segments_end(end, gap, theta):
    """The walk's leaves: the same pair, every cell opened (no cell of these eight
    points is small enough beside its distance to be taken whole at 1e-3; the sum is
    the direct one without the infront neighbour's straight segment)."""
    import torch

    from qvort_b200 import adjoint as A
    from qvort_b200 import lib as L

    for seed in range(4):
        w, _ = _system(end, gap, seed)
        w.params.update(velocity="Tree", tree_theta=1e-3 * theta)
        # only the target's velocity: its own neighbours' segments are straight on
        # with it, and the triangle's are not its neighbours
        ubar = np.zeros_like(w.x)
        ubar[3] = _grid(np.random.default_rng(seed).uniform(-1, 1, 3))
        s = A.FilamentSystem(L.default_params(**w.params), w.infront, w.behind)
        x = torch.tensor(w.x, device="cuda", requires_grad=True)
        (g,) = torch.autograd.grad(A.velocity(x, s), x, torch.tensor(ubar, device="cuda"))
        s.close()
        og = _sum_vjp(w, ubar, "open")
        # the segment from the infront neighbour on is the walk's to skip
        f = w.infront - 1
        G = LD(w.params["quant_circ"]) / (4 * LD(np.pi))
        j = f[3]
        for t in (3, j, f[j]):
            for c in range(3):
                y = w.x.astype(CD)
                y[t, c] += CD(1e-40j)
                v = G * _segment(y[j] - y[3], y[f[j]] - y[3])
                og[t, c] -= float((v * ubar[3]).sum().imag / LD(1e-40))
        assert np.abs(g.cpu().numpy() - og).max() <= TOL * np.abs(og).max()


@pytest.mark.parametrize("images", [False, True])
@pytest.mark.parametrize("bc", ["open", "openxy", "openx", "periodic"])
@pytest.mark.parametrize("gap", [0.07, 0.2, 0.5])
@pytest.mark.parametrize("end", [1, 2])
def test_jacobian_at_a_point_near_a_segments_end(end, gap, bc, images):
    from qvort_b200 import lib as L

    for seed in range(4):
        w, P = _system(end, gap, seed)
        x, f = w.x[:3], w.infront[:3] - 1
        c = L.Context(L.default_params(**dict(w.params, boundary=bc)))
        c.set_points(x, w.infront[:3], w.behind[:3])
        P = w.x[3]
        J = c.field_velocity(P[None], images)[1][0]
        c.close()
        G = LD(w.params["quant_circ"]) / (4 * LD(np.pi))
        oJ = np.empty((3, 3))
        for k in range(3):
            p = P.astype(CD)
            p[k] += CD(1e-40j)
            v = 0
            for sh in _shifts(bc) if images else [np.zeros(3, LD)]:
                v = v + G * _segment(x + sh - p, x[f] + sh - p).sum(0)
            oJ[:, k] = (v.imag / LD(1e-40)).astype(np.float64)
        assert np.abs(J - oJ).max() <= TOL * np.abs(oJ).max()
