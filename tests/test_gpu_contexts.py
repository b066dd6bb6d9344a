"""GPU tests of what contexts of one process owe each other and their caller:
launch attributes that belong to the process, and results and memory that belong
to the caller."""
import numpy as np
import pytest

from qvort_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _deep(depth, seed=0):
    """A ring and a triangle with one side of 0.1 x 2^-depth: a tree a few levels
    on either side of `depth` levels deep."""
    w = W.ring(40, 0.01, 1e-5, seed=seed)
    a = np.array([0.0323, 0.0211, 0.0157])
    tri = np.array([a, a + 0.1 * 2.0 ** -depth * np.array([0.9, 0.7, 0.8]), a + [1e-3, -2e-3, 1e-3]])
    w.x = np.concatenate([w.x, tri])
    w.infront = np.concatenate([w.infront, [42, 43, 41]]).astype(np.int32)
    w.behind = np.concatenate([w.behind, [43, 41, 42]]).astype(np.int32)
    w.params = dict(w.params, boundary="periodic", velocity="Tree", tree_theta=0.4, box_size=0.1)
    return w


def _ctx(w, **kw):
    from qvort_b200 import lib as L

    c = L.Context(L.default_params(**dict(w.params, **kw)))
    c.set_points(w.x, w.infront, w.behind)
    return c


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_deep_trees_in_several_contexts(precision):
    """Walks and searches whose stacks need more shared memory than a launch has by
    default: the size a kernel may ask for belongs to the process, so a context
    with a shallower tree must not take it from one with a deeper tree."""
    a, b = (_ctx(_deep(d), precision=precision) for d in (44, 34))
    ua, ub = a.velocity()[0], b.velocity()[0]
    pts = np.random.default_rng(0).uniform(-0.05, 0.05, (40, 3))
    fa = a.field_velocity_tree(pts)[0]
    ca = a.closest()
    fb, cb = b.field_velocity_tree(pts)[0], b.closest()
    for c, u, f, s in ((a, ua, fa, ca), (b, ub, fb, cb), (a, ua, fa, ca)):
        assert np.array_equal(c.velocity()[0], u)
        assert np.array_equal(c.field_velocity_tree(pts)[0], f)
        assert all(np.array_equal(p, q) for p, q in zip(c.closest(), s))


def test_deep_trees_in_several_batches():
    """The same for batches, with the largest blocks a batch can be given."""
    from qvort_b200 import lib as L

    def batch(depth):
        w = _deep(depth)
        p = L.default_params(**dict(w.params, boundary="open", precision="mixed"))
        return L.Batch(p, [(w.x, w.infront, w.behind)], ["Tree"], [1e-12])

    a, b = batch(44), batch(20)
    ua = a.velocity()
    for t in (a, b, a):
        t.set_config(8, 1, 0)
        t.velocity()
    assert np.array_equal(a.velocity(), ua)


def test_velocity_device_leaves_the_array_alone_on_a_singularity():
    import torch

    from qvort_b200 import lib as L

    w = W.ring(40, 0.01, 1e-5)
    w.x[20] = w.x[3] + [1e-16, 0.0, 0.0]  # not neighbours, within epsilon
    c = _ctx(w, velocity="Tree", tree_theta=0.4, precision="fp64")
    u = torch.full((w.n, 3), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with pytest.raises(L.QvError):
        c.velocity_device(u.data_ptr())
    assert (u == 7.0).all()
    w.x[20] = W.ring(40, 0.01, 1e-5).x[20]
    c.set_points(w.x, w.infront, w.behind)
    c.velocity_device(u.data_ptr())
    assert np.array_equal(u.cpu().numpy(), c.velocity()[0])


@pytest.mark.parametrize("bc", ["open", "periodic"])
@pytest.mark.parametrize("rk3", [0, 1])
@pytest.mark.parametrize("velocity", ["BS", "Tree"])
def test_profiled_steps_report_ghosts_and_local_term(velocity, rk3, bc):
    """Each phase of a step has its own time, and profiling changes no bit."""
    w = W.ring(300, 0.01, 1e-5, seed=1)
    kw = dict(velocity=velocity, tree_theta=0.4 if velocity == "Tree" else 0.0, boundary=bc,
              runge_kutta=rk3, precision="fp64")
    a, b = _ctx(w, **kw), _ctx(w, **kw)
    a.profile(True)
    for k in range(1, 5):
        a.step(k)
        b.step(k)
    t = a.phase_times()
    for ph in ("ghosts", "local", "nonlocal", "update", "wrap"):
        assert t[ph] > 0.0, ph
    assert all(np.array_equal(p, q) for p, q in zip(a.get_points(), b.get_points()))


def _used():
    import torch

    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


@pytest.mark.parametrize("tree,m", [(False, 3_000_000), (True, 6_000_000)])
def test_field_calls_give_large_buffers_back(tree, m):
    """A context keeps at most 256 MB for its field points between calls."""
    w = W.ring(5, 0.01, 1e-5)
    c = _ctx(w, velocity="Tree" if tree else "BS", tree_theta=0.4 if tree else 0.0,
             precision="fp64")
    few = np.random.default_rng(1).uniform(-0.05, 0.05, (100, 3))
    call = c.field_velocity_tree if tree else c.field_velocity
    u = call(few)[0]
    used = _used()
    pts = np.broadcast_to(few, (m // 100, 100, 3)).reshape(m, 3)
    v = call(pts)[0]
    assert np.array_equal(v.reshape(-1, 100, 3), np.broadcast_to(u, (m // 100, 100, 3)))
    assert _used() - used <= (256 << 20) + (4 << 20)  # and the allocator's granularity


@pytest.mark.parametrize("m", [1_048_575, 1_048_577, 1_050_000])
def test_field_points_in_several_launches(m):
    """Direct field points either side of the largest launch: each has the value and
    the Jacobian of a call of its own."""
    w = W.ring(33, 0.01, 1e-5)
    c = _ctx(w, precision="fp64")
    rng = np.random.default_rng(m)
    pts = rng.uniform(-0.05, 0.05, (m, 3))
    u, J = c.field_velocity(pts)
    at = np.unique(np.r_[0, rng.integers(0, m, 200), np.arange(1_048_570, m)[:40], m - 1])
    v, K = c.field_velocity(pts[at])
    # a small call cuts the sources in chunks: sums in another order
    assert np.abs(u[at] - v).max() <= 1e-13 * np.abs(v).max()
    assert np.abs(J[at] - K).max() <= 1e-13 * np.abs(K).max()


@pytest.mark.parametrize("small,large,pair", [(9000, 0, False), (8000, 800, False),
                                              (3000, 3000, True), (0, 2900, False),
                                              (0, 3000, True)])
def test_batched_walk_takes_pairs_where_they_save_items(small, large, pair):
    """Systems of at most 32 points gain nothing from items of 64 targets, whatever
    their number: the choice counts the items saved (160 per SM, 23,680 on 148)."""
    from qvort_b200 import lib as L

    w, v = W.ring(32, 0.01, 1e-5), W.ring(64, 0.01, 1e-5)
    ws = [(w.x, w.infront, w.behind)] * small + [(v.x, v.infront, v.behind)] * large
    b = L.Batch(L.default_params(**dict(w.params, velocity="Tree", tree_theta=0.4,
                                        precision="mixed")), ws, ["Tree"] * len(ws),
                [1e-9] * len(ws))
    assert b.stats()["items"] == 8 * (small + (1 if pair else 2) * large)


def test_launch_count_of_a_tree_gradient():
    """A tree of at most 585 nodes needs one moment kernel, a larger one two."""
    import torch

    from qvort_b200 import lib as L

    n = []
    for m in (64, 2000):
        w = W.ring(m, 0.01, 1e-5)
        c = L.Context(L.default_params(**dict(w.params, velocity="Tree", tree_theta=0.4,
                                              precision="fp64")), stream=1)
        c.set_points(w.x, w.infront, w.behind)
        c.velocity()
        nodes = c.tree_info()[0]
        assert (nodes <= 585) == (m == 64)
        x, y = (torch.ones(m, 3, dtype=torch.float64, device="cuda") for _ in range(2))
        c.velocity_vjp(x.data_ptr(), y.data_ptr())
        k = c.counters()["launches"]
        c.velocity_vjp(x.data_ptr(), y.data_ptr())
        n.append(c.counters()["launches"] - k)
    assert n[1] == n[0] + 1

@pytest.mark.parametrize("n", [5, 1000, 100_000])
def test_velocity_device_writes_its_array_and_nothing_else(n):
    """Into the middle of a device array (copied by a kernel) and of a pinned one (by the
    runtime): the velocities of the host call, and nothing around them."""
    import torch

    w = W.ring(n, 0.01, 1e-5)
    c = _ctx(w, velocity="LIA" if n > 5000 else "BS", precision="fp64")
    u = c.velocity()[0]
    for kw in (dict(device="cuda"), dict(pin_memory=True)):
        a = torch.full((3 * n + 9,), 7.0, dtype=torch.float64, **kw)
        torch.cuda.synchronize()
        c.velocity_device(a.data_ptr() + 8 * 4)
        a = a.cpu().numpy()
        assert np.array_equal(a[4:4 + 3 * n].reshape(n, 3), u)
        assert (a[:4] == 7.0).all() and (a[4 + 3 * n:] == 7.0).all()
    # an address that is no multiple of eight: the runtime's copy as well
    b = torch.zeros(24 * n + 4, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    c.velocity_device(b.data_ptr() + 4)
    assert np.array_equal(b.cpu().numpy()[4:].view(np.float64).reshape(n, 3), u)
