"""GPU test of the opening decisions of the Barnes-Hut gradient in shifted images:
they are the velocity's, also for cells so small that the rounding of a shifted
coordinate is visible in their distance."""
import numpy as np
import pytest

from qvort_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _distance(x, cent, s):
    v = x - (cent + s)
    return np.sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2])


@pytest.mark.parametrize("seed", range(4))
def test_gradient_opens_the_cells_the_velocity_opens(seed):
    """A cell of two points (width box x 2^-24) just inside one face and a target just
    inside the opposite one, so near the cell's opening radius that (x - s) - c and
    x - (c + s) fall on either side of it.  The velocity takes the second: the cell
    is far.  Moving the target off by 1e-3 of the distance keeps it far and changes
    nothing by more than a few times that; with the cell opened the velocity and its
    gradient differ by orders of magnitude."""
    import torch

    from qvort_b200 import adjoint as A
    from qvort_b200 import lib as L

    box, theta, depth = 0.125, 0.5, 24  # x - s and c + s round at this box
    width = box / 2 ** depth
    rng = np.random.default_rng(seed)
    # the two points: opposite octants of one cell of that depth, beside the face +x
    lo = np.array([2 ** depth - 1, 2 ** (depth - 1) + 12345, 2 ** (depth - 1) + 6789 + seed]) * width - box / 2
    a = lo + width * rng.uniform(0.1, 0.4, 3)
    b = lo + width * rng.uniform(0.6, 0.9, 3)
    cent = (a + b) / 2.0
    s = np.array([-box, 0.0, 0.0])
    rc = width / theta

    def far(x):
        return width / _distance(x, cent, s) < theta

    # a target at 0.9 of the radius along x, the rest along y, just outside the radius
    x = np.array([(cent[0] - box) + 0.9 * rc, cent[1], cent[2]])
    found = None
    for k in range(400):
        x[0] = np.nextafter(x[0], 1.0)
        if not x[0] > -box / 2:
            continue
        vf, vb = x[0] - (cent[0] + s[0]), (x[0] - s[0]) - cent[0]
        if not vb < vf:
            continue
        # rc^2 lies between the two squared distances, nearer to the velocity's
        y = np.sqrt(rc * rc * (1 + 1e-11) - vf * vf)
        p = x.copy()
        for _ in range(2000):
            p[1] = cent[1] + y
            if far(p):
                break
            y = np.nextafter(y, 1.0) + 1e-22
        d2b = vb * vb + (p[1] - cent[1]) ** 2
        if far(p) and d2b < rc * rc * (1 - 5e-11):
            found = p
            break
    assert found is not None
    moved, inside = found.copy(), found.copy()
    moved[1] = cent[1] + 1.001 * (found[1] - cent[1])
    inside[1] = cent[1] + 0.9 * (found[1] - cent[1])
    assert far(found) and far(moved) and not far(inside)

    def run(p):
        pts = np.array([a, b, [0.01, 0.02, 0.015],
                        p, p + [0.003, 0.004, 0.002], p + [0.006, -0.003, 0.004],
                        p + [0.004, -0.006, -0.005], p + [0.002, -0.002, -0.006]])
        inf = np.array([2, 3, 1, 5, 6, 7, 8, 4], np.int32)
        beh = np.array([3, 1, 2, 8, 4, 5, 6, 7], np.int32)
        q = L.default_params(boundary="periodic", velocity="Tree", tree_theta=theta, box_size=box,
                             deriv_order=2, quant_circ=W.GAMMA_HE4, corea=W.CORE_A,
                             precision="fp64", tree_extra_correction=0)
        c = L.Context(q)
        c.set_points(pts, inf, beh)
        c.ghosts()
        c.build_tree()
        t = c.tree_export()
        k = np.flatnonzero((t["depth"] == depth) & (t["pcount"] == 2))
        assert len(k) == 1 and np.array_equal(t["cent"][k[0]], cent) and t["width"][k[0]] == width
        c.close()
        sy = A.FilamentSystem(q, inf, beh)
        x = torch.tensor(pts, device="cuda", requires_grad=True)
        u = A.velocity(x, sy)
        ubar = torch.zeros_like(x)
        ubar[3] = torch.tensor([0.3, -0.7, 0.5], dtype=torch.float64)
        (g,) = torch.autograd.grad(u, x, ubar)
        sy.close()
        return u.detach().cpu().numpy()[3], g.cpu().numpy()[3]

    (u0, g0), (u1, g1), (u2, g2) = run(found), run(moved), run(inside)
    assert np.abs(u0 - u1).max() <= 0.05 * np.abs(u1).max()   # both far
    assert np.abs(u0 - u2).max() >= 0.5 * np.abs(u0).max()    # opened: another velocity
    assert np.abs(g0 - g1).max() <= 0.05 * np.abs(g1).max()
