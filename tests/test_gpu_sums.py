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


def _direct_vjp(w, ubar, bc):
    """x_bar of the BS arm by torch autograd: local term (second order) and the
    direct sum over images, without the pairs whose target lies exactly on the
    segment's line (they are left out of the gradient)."""
    import torch

    p = O.params(**dict(w.params, boundary=bc))
    x = torch.tensor(w.x, requires_grad=True)
    inf, beh = torch.tensor(w.infront).long() - 1, torch.tensor(w.behind).long() - 1
    g = O.ghosts(p, w.x, w.infront, w.behind)
    gi = x[inf] + (torch.tensor(g[0]) - x[inf]).detach()
    gb = x[beh] + (torch.tensor(g[1]) - x[beh]).detach()
    i, b = (x - gi).norm(dim=1, keepdim=True), (x - gb).norm(dim=1, keepdim=True)
    s1 = (b * gi + (i - b) * x - i * gb) / (2 * b * i)
    s2 = 2 * (gi / (i * (i + b)) - x / (i * b) + gb / (b * (i + b)))
    G = p.quant_circ / (4 * np.pi)
    loss = (G * torch.log(1.21 / p.corea * torch.sqrt(i * b)) * torch.linalg.cross(s1, s2)
            * torch.tensor(ubar)).sum()
    n = w.n
    ax = {"open": (0, 0, 0), "openxy": (0, 0, 1), "openx": (0, 1, 1), "periodic": (1, 1, 1)}[bc]
    for a in range(-ax[0], ax[0] + 1):
        for c in range(-ax[1], ax[1] + 1):
            for d in range(-ax[2], ax[2] + 1):
                sh = torch.tensor([a, c, d], dtype=torch.float64) * p.box_size
                skip = torch.arange(n)[None] == beh[:, None]
                if (a, c, d) == (0, 0, 0):
                    skip = skip | torch.eye(n, dtype=torch.bool)
                r1 = (x + sh)[None] - x[:, None]
                s = (gi - x)[None].expand_as(r1)
                skip = skip | (torch.linalg.cross(r1, s).detach() == 0).all(-1)
                r1 = torch.where(skip[..., None], torch.ones_like(r1), r1)
                s = torch.where(skip[..., None], torch.tensor([1.0, 0.0, 0.0]).double(), s)
                r2, cr = r1 + s, torch.linalg.cross(r1, s)
                A, B, D = r1.norm(dim=-1), r2.norm(dim=-1), (r1 * r2).sum(-1)
                den = torch.where(D < 0, (cr * cr).sum(-1) / torch.where(D < 0, A * B - D, 1.0),
                                  A * B + D)
                f = (A + B) / (A * B * den) * (~skip)
                loss = loss + (G * f[..., None] * cr * torch.tensor(ubar)[:, None]).sum()
    return torch.autograd.grad(loss, x)[0].numpy()


def _vjp(w, ubar, bc):
    import torch

    from qvort_b200 import adjoint as A
    from qvort_b200 import lib as L

    s = A.FilamentSystem(L.default_params(**dict(w.params, boundary=bc, precision="fp64")),
                         w.infront, w.behind)
    x = torch.tensor(w.x, device="cuda", requires_grad=True)
    (g,) = torch.autograd.grad(A.velocity(x, s), x, torch.tensor(ubar, device="cuda"))
    s.close()
    return g.cpu().numpy()


@pytest.mark.parametrize("bc", ["open", "openxy", "openx", "periodic"])
@pytest.mark.parametrize("n", [5, 31, 33, 128, 129, 260])
def test_direct_vjp_at_tile_and_chunk_edges(n, bc):
    """Both ends' gradients of every pair.  Each gradient is a difference of
    terms larger by at most |d|/|s| < 1e4 (see above): 1e-11 of the largest."""
    w = _ring_pair(n)
    ubar = np.random.default_rng(n).normal(0.0, 0.1, w.x.shape)
    g, og = _vjp(w, ubar, bc), _direct_vjp(w, ubar, bc)
    assert np.abs(g - og).max() <= 1e-11 * np.abs(og).max()


@pytest.mark.parametrize("bc", ["open", "periodic"])
def test_direct_vjp_near_and_on_a_segments_line(bc):
    """A target beside the middle of another filament's segment (obtuse angle
    between its ends), a square of axis-parallel sides whose points lie exactly
    on one another's lines, and a planar ring."""
    w = W.ring(24, 0.01, 0.0, seed=1)          # exactly in z = 0
    h = 0.0078125
    t = np.arange(4)[:, None] * h
    o = np.zeros((4, 1))
    sq = np.concatenate([np.hstack([t, o, o]), np.hstack([o + 4 * h, t, o]),
                         np.hstack([4 * h - t, o + 4 * h, o]), np.hstack([o, 4 * h - t, o])])
    sq = sq + [-0.03125, -0.03125, 0.015625]
    k = w.n
    mid = 0.5 * (w.x[3] + w.x[4]) + [0.0, 0.0, 2e-5]
    near = np.array([mid, mid + [0.004, 0.001, 0.003], mid + [-0.002, 0.004, 0.005],
                     mid + [0.001, -0.003, 0.002], mid + [0.003, 0.003, 0.006]])
    m = len(sq)
    x = np.concatenate([w.x, sq, near])
    inf = np.concatenate([w.infront, k + 1 + (np.arange(m) + 1) % m,
                          k + m + 1 + (np.arange(5) + 1) % 5]).astype(np.int32)
    beh = np.concatenate([w.behind, k + 1 + (np.arange(m) - 1) % m,
                          k + m + 1 + (np.arange(5) - 1) % 5]).astype(np.int32)
    v = W.Workload("lines", x, inf, beh, w.params)
    ubar = np.random.default_rng(3).normal(0.0, 0.1, x.shape)
    g, og = _vjp(v, ubar, bc), _direct_vjp(v, ubar, bc)
    assert np.isfinite(g).all()
    # the near pair's 1 + cos is about 1e-3 of 1: its digits cost another 1e3
    assert np.abs(g - og).max() <= 1e-9 * np.abs(og).max()


@pytest.mark.parametrize("bc", ["open", "openxy", "openx", "periodic"])
@pytest.mark.parametrize("m", [1, 31, 33, 129, 700, 66000])
def test_field_velocity_tree_at_group_and_slab_edges(m, bc):
    """Points per warp, cells of their Morton order and points per launch at their
    edges, points outside the box and on a filament among them.  The sums are
    FP64 in another order than the oracle's: its far cells and leaves agree to a
    few ulp of each term, the terms to 1e3 of the sum: 1e-12 of the largest."""
    w = W.random_rings(4, 0.006, 0.012, 5e-4, 0.1, seed=m)
    rng = np.random.default_rng(m)
    pts = rng.uniform(-0.05, 0.05, (m, 3))
    pts[::7] = rng.uniform(-0.08, 0.08, pts[::7].shape)
    pts[::11] = w.x[rng.integers(0, w.n, len(pts[::11]))]
    c = _ctx(w, boundary=bc, velocity="Tree", tree_theta=0.4, precision="fp64")
    u, ev = c.field_velocity_tree(pts)
    pick = np.arange(m) if m < 1000 else np.unique(np.r_[rng.integers(0, m, 300), 65535, 65536])
    p = O.params(**dict(w.params, boundary=bc, velocity="Tree", tree_theta=0.4))
    g = O.ghosts(p, w.x, w.infront, w.behind)
    tree = O.Tree(p, w.x, g[0], w.infront)
    ou, oev = O.field_velocity_tree(p, tree, pts[pick])
    tree.close()
    if m < 1000:
        assert ev == oev
    assert np.array_equal(np.isnan(u[pick]), np.isnan(ou))
    ok = ~np.isnan(ou).any(axis=1)
    if ok.any():
        assert np.abs(u[pick] - ou)[ok].max() <= 1e-12 * np.abs(ou[ok]).max()


@pytest.mark.parametrize("bc", ["open", "openxy", "openx", "periodic"])
@pytest.mark.parametrize("n", [5, 31, 33, 64, 129, 260])
def test_tree_velocity_and_vjp_at_group_edges(n, bc):
    """FP64 Barnes-Hut velocity and its gradient with the opened cells held, at
    the edges of the walks' target groups, against torch autograd over the same
    cells (perf/cases.py): both in FP64, 1e-11 of the largest as above."""
    import torch

    from perf import cases as P
    from qvort_b200 import adjoint as A
    from qvort_b200 import lib as L

    w = _ring_pair(n)
    w.params = dict(w.params, boundary=bc, velocity="Tree", tree_theta=0.45, precision="fp64",
                    deriv_order=2)
    ubar = np.random.default_rng(n).normal(0.0, 0.1, w.x.shape)
    ou, og = (t.detach().cpu().numpy() for t in P._tree_u(w, torch.tensor(ubar, device=P._dev())))
    s = A.FilamentSystem(L.default_params(**w.params), w.infront, w.behind)
    x = torch.tensor(w.x, device="cuda", requires_grad=True)
    u = A.velocity(x, s)
    (g,) = torch.autograd.grad(u, x, torch.tensor(ubar, device="cuda"))
    s.close()
    assert np.abs(u.detach().cpu().numpy() - ou).max() <= 1e-11 * np.abs(ou).max()
    assert np.abs(g.cpu().numpy() - og).max() <= 1e-11 * np.abs(og).max()


@pytest.mark.parametrize("n", [1, 5, 31, 33, 64, 130, 4095, 4096, 4097, 4101])
def test_pclose_at_split_edges_with_ties_and_empty_slots(n):
    """The all-pairs search on either side of its split (one target per warp, four
    beyond 4096 slots), on points of a coarse lattice -- most least distances
    are ties, decided by the slot order -- with empty slots: bit for bit."""
    rng = np.random.default_rng(n)
    x = rng.integers(-6, 7, (n, 3)) * 0.0078125
    inf, beh = (np.arange(n) + 1) % n + 1, (np.arange(n) - 1) % n + 1
    if n > 40:  # drop a few points from the chain
        for i in range(7, n - 3, 11):
            inf[beh[i] - 1], beh[inf[i] - 1] = inf[i], beh[i]
            inf[i] = beh[i] = 0
    w = W.Workload("lattice", x, inf.astype(np.int32), beh.astype(np.int32),
                   dict(boundary="open", velocity="LIA", tree_theta=0.0, box_size=0.1, dt=1e-7,
                        delta=5e-4))
    seed = rng.integers(0, n + 1, n).astype(np.int32)
    c = _ctx(w)
    c.set_closest(seed)
    cl, cd = c.closest()
    ocl, ocd = O.pclose(x, w.infront, w.behind, seed)
    act = inf != 0
    assert np.array_equal(cl, ocl)
    assert np.array_equal(cd[act], ocd[act])


@pytest.mark.parametrize("bc", ["open", "periodic"])
@pytest.mark.parametrize("n", [4095, 4096, 4097])
def test_direct_fp64_either_side_of_the_small_sum(n, bc):
    """The last sizes with a block per target and the first with tiles, on 64 of
    the targets (1e-11 as above); the evaluation count needs the active count."""
    w = _ring_pair(n)
    u, _, _, ev = _ctx(w, boundary=bc, precision="fp64").velocity()
    assert ev == n * n * (27 if bc == "periodic" else 1)
    at = np.unique(np.random.default_rng(n).integers(0, n, 64))
    x = w.x[at]
    p = O.params(**dict(w.params, boundary=bc))
    g = O.ghosts(p, w.x, w.infront, w.behind)
    ou = O.velocity(p, w.x, w.infront, w.behind, g, nthreads=8)[0]
    assert len(x) and np.abs(u - ou)[at].max() <= 1e-11 * np.abs(ou[at]).max()


@pytest.mark.parametrize("bc", ["open", "openx", "periodic"])
@pytest.mark.parametrize("velocity,order", [("BS", 2), ("BS", 4), ("LIA", 4), ("Off", 2)])
def test_ghosts_and_local_term_in_one_launch_equal_two(velocity, order, bc):
    """A velocity that gathers its own ghosts takes them and the local term in one
    kernel, one on given ghosts the local term alone: the same bits, and the
    oracle's ghosts."""
    w = _ring_pair(301)
    kw = dict(velocity=velocity, deriv_order=order, boundary=bc, precision="fp64")
    a, b = _ctx(w, **kw), _ctx(w, **kw)
    b.ghosts()
    ua, la, *_ = a.velocity()
    ub, lb, *_ = b.velocity()
    assert np.array_equal(ua, ub) and np.array_equal(la, lb)
    og = O.ghosts(O.params(**dict(w.params, boundary=bc)), w.x, w.infront, w.behind)
    for g, h, o in zip(a.get_ghosts(), b.get_ghosts(), og):
        assert np.array_equal(g, h) and np.array_equal(g, o)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 127, 128, 129, 4095, 4097, 8190, 65535, 65536, 65537])
def test_active_list_at_its_edges(n):
    """The ordered list of the active slots (one block up to 65,536 slots): points
    with empty slots among them keep their order -- a mixed direct sum over the
    list gives each filament's own velocity wherever its slots lie."""
    from qvort_b200 import lib as L

    m = min(n, 12)
    w = W.ring(m, 0.01, 1e-5, seed=2) if m > 4 else None
    rng = np.random.default_rng(n)
    x = rng.uniform(-0.04, 0.04, (n, 3))
    inf, beh = np.zeros(n, np.int32), np.zeros(n, np.int32)
    at = np.sort(rng.choice(n, m, replace=False))
    at[-1] = n - 1
    if m > 4:
        x[at] = w.x
        inf[at], beh[at] = at[w.infront - 1] + 1, at[w.behind - 1] + 1
    kw = dict(boundary="open", velocity="BS", tree_theta=0.0, box_size=0.1, precision="mixed",
              quant_circ=W.GAMMA_HE4, corea=W.CORE_A)
    c = L.Context(L.default_params(**kw))
    c.set_points(x, inf, beh)
    u, _, _, ev = c.velocity()
    assert ev == (m * m if m > 4 else 0)
    if m > 4:
        d = L.Context(L.default_params(**kw))
        d.set_points(w.x, w.infront, w.behind)
        assert np.array_equal(u[at], d.velocity()[0])


def test_tree_moments_at_the_kernels_node_sizes():
    """Nodes of the sizes where one moment kernel hands over to the next (8 | 9
    points, 32 | 33, 512 | 513) and around a warp's 32-point pieces: every node's
    moments bit for bit the oracle's."""
    from qvort_b200 import lib as L

    sizes = [1, 2, 8, 9, 31, 32, 33, 64, 65, 127, 128, 129, 511, 512, 513, 640]
    rng = np.random.default_rng(9)
    cells = rng.permutation(64)[:len(sizes)]  # one of the 4^3 cells of level 2 each
    x = []
    for m, q in zip(sizes, cells):
        corner = np.array([q % 4, q // 4 % 4, q // 16]) * 0.025 - 0.05
        x.append(corner + rng.uniform(0.001, 0.024, (m, 3)))
    x = np.concatenate(x)[rng.permutation(sum(sizes))]
    n = len(x)
    k = np.arange(n)
    inf, beh = ((k + 1) % n + 1).astype(np.int32), ((k - 1) % n + 1).astype(np.int32)
    kw = dict(boundary="open", velocity="Tree", tree_theta=0.4, box_size=0.1)
    c = L.Context(L.default_params(**kw))
    c.set_points(x, inf, beh)
    c.ghosts()
    c.build_tree()
    got = c.tree_export()
    p = O.params(**kw)
    want = O.Tree(p, x, O.ghosts(p, x, inf, beh)[0], inf).export()
    assert set(sizes) <= set(got["pcount"][got["depth"] == 2])
    assert set(got) == set(want)
    for name in want:
        np.testing.assert_array_equal(got[name], want[name], err_msg=name)


@pytest.mark.parametrize("seed", [0, 1])
def test_mixed_direct_pairs_equal_the_walks_leaf_pairs(seed):
    """The direct sum's pair term (one branch for cos >= 0) has the bits of the
    walk's leaf pair (no branch): a point and a triangle whose corners the tree
    visits in slot order, seen under every angle, near its ends and from afar."""
    from qvort_b200 import lib as L

    rng = np.random.default_rng(seed)
    A, B, C = np.array([[0.005, 0.006, 0.004], [0.03, 0.011, 0.02], [0.04, 0.03, 0.045]])
    far = rng.uniform(-0.045, 0.045, (60, 3))
    near = A + rng.uniform(-1.0, 1.0, (30, 3)) * 10.0 ** rng.uniform(-7, -3, (30, 1))
    line = A + rng.uniform(-0.1, 1.1, (30, 1)) * (B - A) + rng.uniform(-1e-5, 1e-5, (30, 3))
    P = np.concatenate([far, near, line])
    cos = np.einsum("ij,ij->i", A - P, B - P)
    assert (cos > 0).any() and (cos < 0).any()
    inf, beh = np.array([2, 1, 4, 5, 3], np.int32), np.array([2, 1, 5, 3, 4], np.int32)
    ws = [(np.array([p, [-0.04, -0.03, 0.02], A, B, C]), inf, beh) for p in P]
    kw = dict(boundary="open", box_size=0.1, precision="mixed", quant_circ=W.GAMMA_HE4,
              corea=W.CORE_A, tree_theta=1e-3)
    n = len(ws)
    u = {v: L.Batch(L.default_params(**kw, velocity="Tree"), ws, [v] * n, [1e-7] * n).velocity()
         for v in ("BS", "Tree")}
    assert np.array_equal(u["BS"][::5], u["Tree"][::5])
    for k in range(0, n, 17):
        c = L.Context(L.default_params(**dict(kw, velocity="BS", tree_theta=0.0)))
        c.set_points(*ws[k])
        assert np.array_equal(c.velocity()[0][0], u["BS"][5 * k])
        c.close()


@pytest.mark.parametrize("n", [43_690, 43_691, 60_000])
def test_large_results_into_fresh_and_offset_arrays(n):
    """Results around and above 1 MB (the pages of larger arrays are made before the
    copy): a new array, a used one and an unaligned slice get the same values, and
    nothing outside the slice is written."""
    from qvort_b200 import lib as L

    w = W.ring(n, 0.01, 0.0)
    c = L.Context(L.default_params(**dict(w.params, velocity="LIA", precision="fp64")))
    c.set_points(w.x, w.infront, w.behind)
    u = c.velocity()[0]
    x0, u0 = c.get_points()
    assert np.array_equal(x0, w.x) and np.array_equal(u0, u)
    pad = np.full(2 * 3 * n + 1111, 7.0)
    xs, us = pad[5:5 + 3 * n].reshape(n, 3), pad[1000 + 3 * n:1000 + 6 * n].reshape(n, 3)
    c.get_points(xs, us)
    assert np.array_equal(xs, x0) and np.array_equal(us, u0)
    assert (pad[:5] == 7).all() and (pad[5 + 3 * n:1000 + 3 * n] == 7).all()
    assert (pad[1000 + 6 * n:] == 7).all()
    b = L.Batch(L.default_params(**dict(w.params, precision="mixed", velocity="Tree",
                                        tree_theta=0.4)),
                [(w.x, w.infront, w.behind)], ["Tree"], [1e-9])
    assert np.array_equal(b.get_points()[0], w.x)
    v = b.velocity()
    assert np.array_equal(b.get_points()[1], v)


def test_batched_walk_with_two_targets_a_lane_equals_one():
    """A batch large enough for walk items of 64 targets (71,040 items of 32 on 148
    SMs): systems around multiples of 32 and 64 points, each repeated, have bit for
    bit the velocities of the same systems in a small batch, and the same steps."""
    from qvort_b200 import lib as L

    sizes = [5, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 1000]
    ws = [W.ring(m, 0.01 + 1e-5 * k, 1e-5, seed=k) for k, m in enumerate(sizes)]
    reps = 160
    p = L.default_params(boundary="open", velocity="Tree", tree_theta=0.4, box_size=0.1,
                         precision="mixed", quant_circ=W.GAMMA_HE4, corea=W.CORE_A)

    def batch(r):
        m = len(ws) * r
        return L.Batch(p, [(w.x, w.infront, w.behind) for w in ws] * r, ["Tree"] * m, [1e-9] * m)

    small, large = batch(1), batch(reps)
    assert 8 * reps * sum(-(-m // 32) for m in sizes) >= 71_040
    # one item per 64 targets of a system and root child
    assert large.stats()["items"] == 8 * reps * sum(-(-m // 64) for m in sizes)
    assert small.stats()["items"] == 8 * sum(-(-m // 32) for m in sizes)
    us, ul = small.velocity(), large.velocity()
    assert np.array_equal(ul.reshape(reps, -1, 3), np.broadcast_to(us, (reps, *us.shape)))
    small.step(3)
    large.step(3)
    xs, xl = small.get_points()[0], large.get_points()[0]
    assert np.array_equal(xl.reshape(reps, -1, 3), np.broadcast_to(xs, (reps, *xs.shape)))
