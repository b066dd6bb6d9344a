"""GPU tests of the FP64 pair sums at the sizes where their splits change:
edges of target tiles and source chunks, one and two tiles, every boundary.

Tolerance: the oracle's direct form takes (2c+b)/sqrt(a+b+c) - b/sqrt(a), which
loses a factor |d|/|s| (box diagonal over segment, below 1e4 for these
systems) of FP64's 1.1e-16 per term: 1e-11 of the largest velocity covers it.
"""
import numpy as np
import pytest

from oracle import oracle as O
from qvort_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _ctx(w, **kw):
    from qvort_b200 import lib as L

    c = L.Context(L.default_params(**dict(w.params, **kw)))
    c.set_points(w.x, w.infront, w.behind)
    return c


def _oracle_velocity(w, **kw):
    p = O.params(**dict(w.params, **kw))
    g = O.ghosts(p, w.x, w.infront, w.behind)
    return O.velocity(p, w.x, w.infront, w.behind, g)


def _ring_pair(n):
    """n points on two rings (one below 10 points), off the origin and tilted."""
    m = n if n < 10 else n // 2
    w = W.ring(m, 0.01, 1e-5, seed=n)
    if m < n:
        v = W.ring(n - m, 0.013, 1e-5, seed=n + 1)
        w.x = np.concatenate([w.x, v.x[:, [2, 0, 1]] + [0.004, 0.0, 0.003]])
        w.infront = np.concatenate([w.infront, v.infront + m]).astype(np.int32)
        w.behind = np.concatenate([w.behind, v.behind + m]).astype(np.int32)
    w.x = w.x + [0.03, -0.02, 0.01]
    return w


@pytest.mark.parametrize("bc", ["open", "openxy", "openx", "periodic"])
@pytest.mark.parametrize("n", [5, 31, 33, 64, 127, 128, 129, 257, 520])
def test_direct_fp64_at_tile_and_chunk_edges(n, bc):
    w = _ring_pair(n)
    u, _, ubs, _ = _ctx(w, boundary=bc, precision="fp64").velocity()
    ou, _, oubs, *_ = _oracle_velocity(w, boundary=bc)
    assert np.abs(u - ou).max() <= 1e-11 * np.abs(ou).max()
    assert np.abs(ubs - oubs).max() <= 1e-11 * np.abs(oubs).max()


def test_direct_fp64_empty_slots_and_points_on_a_segment():
    """Empty slots take no part, and a point exactly on another segment's line
    (inside it and beyond it) gets nothing from that segment, as in the reference."""
    w = _ring_pair(40)
    # a triangle A-B-C whose side AB has the targets P (its middle) and Q (beyond B)
    A, B, C = [0.0, 0.0, 0.0], [0.0078125, 0.0, 0.0], [0.00390625, 0.015625, 0.0]
    P, Q = [0.00390625, 0.0, 0.0], [0.015625, 0.0, 0.0]
    R = [0.0, 0.0, 0.015625]
    x = np.concatenate([w.x, [A, B, C, P, Q, R], np.full((3, 3), 0.25)])
    k = w.n
    inf = np.concatenate([w.infront, [k + 2, k + 3, k + 1, k + 5, k + 6, k + 4, 0, 0, 0]])
    beh = np.concatenate([w.behind, [k + 3, k + 1, k + 2, k + 6, k + 4, k + 5, 0, 0, 0]])
    v = W.Workload("mixed", x, inf.astype(np.int32), beh.astype(np.int32), w.params)
    for bc in ("open", "periodic"):
        u = _ctx(v, boundary=bc, precision="fp64").velocity()[0]
        ou = _oracle_velocity(v, boundary=bc)[0]
        act = inf != 0
        assert np.isfinite(u[act]).all()
        assert np.abs(u - ou)[act].max() <= 1e-11 * np.abs(ou[act]).max()


def _segment_field(w, pts, bc):
    """Per image, the field at pts of every segment of w, in torch FP64 (autograd)."""
    import torch

    p = O.params(**dict(w.params, boundary=bc))
    gi = O.ghosts(p, w.x, w.infront, w.behind)[0]
    act = w.infront != 0
    x, g = torch.tensor(w.x[act]), torch.tensor(gi[act])
    ax = {"open": (0, 0, 0), "openxy": (0, 0, 1), "openx": (0, 1, 1), "periodic": (1, 1, 1)}[bc]
    sh = [(i, j, k) for i in range(-ax[0], ax[0] + 1) for j in range(-ax[1], ax[1] + 1)
          for k in range(-ax[2], ax[2] + 1)]
    sh.sort(key=lambda t: t != (0, 0, 0))
    for s in sh:
        d = torch.tensor(s, dtype=torch.float64) * p.box_size
        r1, r2 = (x + d)[None] - pts[:, None], (g + d)[None] - pts[:, None]
        a, b, c = r1.norm(dim=-1), r2.norm(dim=-1), (r1 * r2).sum(-1)
        f = (a + b) / (a * b * (a * b + c))
        yield (p.quant_circ / (4 * np.pi)) * (f[..., None] * torch.linalg.cross(r1, r2)).sum(1)


@pytest.mark.parametrize("images", [False, True])
@pytest.mark.parametrize("bc", ["open", "openxy", "openx", "periodic"])
@pytest.mark.parametrize("n,m", [(5, 1), (31, 3), (33, 4), (257, 5), (520, 130)])
def test_field_velocity_and_jacobian_at_split_edges(n, m, bc, images):
    """Points per block, sources per lane and per chunk at their edges.  R1 x R2
    of a segment at distance d cancels to |R1 x s|: a factor d/|s| below 1e4 on
    FP64's 1.1e-16 in the checker, 1e-11 as above."""
    import torch

    w = _ring_pair(n)
    pts = np.random.default_rng(n + m).uniform(-0.045, 0.045, (m, 3))
    u, J = _ctx(w, boundary=bc, precision="fp64", velocity="BS").field_velocity(pts, images)
    P = torch.tensor(pts, requires_grad=True)
    ou, oJ = np.zeros_like(u), np.zeros_like(J)
    for k, v in enumerate(_segment_field(w, P, bc)):
        ou += v.detach().numpy()
        if k == 0 or images:
            for r in range(3):
                oJ[:, r] += torch.autograd.grad(v[:, r].sum(), P, retain_graph=r < 2)[0].numpy()
    assert np.abs(u - ou).max() <= 1e-11 * np.abs(ou).max()
    assert np.abs(J - oJ).max() <= 1e-11 * np.abs(oJ).max()
