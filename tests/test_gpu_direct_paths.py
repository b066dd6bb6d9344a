"""GPU tests of the FP64 direct sum's tile kernel, and of its gradient in several
launches, at the small sizes whose calls take another path by themselves: the edge
tests of test_gpu_sums.py and test_gpu_parity.py, with their tolerances, once more
with the path forced.
"""
import ctypes as C

import numpy as np
import pytest

import test_gpu_parity as P
import test_gpu_sums as S
from oracle import oracle as O
from qvort_b200 import workloads as W

pytestmark = pytest.mark.gpu
BCS = ["open", "openxy", "openx", "periodic"]


@pytest.fixture
def split():
    from qvort_b200 import lib as L

    yield L.test_direct_split
    L.test_direct_split()


@pytest.mark.parametrize("bc", BCS)
@pytest.mark.parametrize("n", [5, 31, 33, 64, 127, 128, 129, 257, 520])
def test_tile_kernel_at_tile_and_chunk_edges(split, n, bc):
    split(0)
    S.test_direct_fp64_at_tile_and_chunk_edges(n, bc)


def test_tile_kernel_with_empty_slots_and_points_on_a_segment(split):
    split(0)
    S.test_direct_fp64_empty_slots_and_points_on_a_segment()


@pytest.mark.parametrize("bc", BCS)
def test_tile_kernel_images_match_oracle(split, bc, nthreads):
    from qvort_b200 import lib as L

    split(0)
    P.test_direct_fp64_images_match_oracle(L, bc, nthreads)


@pytest.mark.parametrize("bc", BCS)
@pytest.mark.parametrize("slots", [0, -1])
@pytest.mark.parametrize("n", [33, 129, 520])
def test_both_kernels_without_allocation(split, n, slots, bc):
    """The entry point on caller's buffers, with empty slots, against the oracle."""
    import torch

    from qvort_b200 import lib as L

    w = S._ring_pair(n)
    x = np.concatenate([w.x, np.full((3, 3), 0.25)])
    inf = np.concatenate([w.infront, [0, 0, 0]]).astype(np.int32)
    beh = np.concatenate([w.behind, [0, 0, 0]]).astype(np.int32)
    v = W.Workload("slots", x, inf, beh, w.params)
    oubs = S._oracle_velocity(v, boundary=bc)[2]
    p = L.default_params(**dict(w.params, boundary=bc, precision="fp64"))
    split(slots)
    d = [torch.tensor(a, device="cuda") for a in (x, inf, beh)]
    out = torch.full((n + 3, 3), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = L.lib().qv_velocity_direct_noalloc(C.byref(p), n + 3, *[t.data_ptr() for t in d],
                                            out.data_ptr(), None)
    assert rc == 0
    got = out.cpu().numpy()
    assert (got[n:] == 0.0).all()
    assert np.abs(got - oubs)[:n].max() <= 1e-11 * np.abs(oubs[:n]).max()


def test_tile_kernel_in_captured_steps_equals_single_steps(split):
    """qv_steps replays the tile kernel from a graph: the bits of qv_step."""
    w = S._ring_pair(300)
    split(0)
    a, b = (S._ctx(w, precision="fp64") for _ in range(2))
    a.steps(1, 6)
    for k in range(1, 7):
        b.step(k)
    assert all(np.array_equal(p, q) for p, q in zip(a.get_points(), b.get_points()))


@pytest.mark.parametrize("bc", BCS)
@pytest.mark.parametrize("n", [31, 33, 128, 129, 260])
def test_gradient_in_several_launches(split, n, bc):
    """32 targets a launch, the last launch short: against autograd, and both ends of
    the near pairs and the pairs on a line as in one launch."""
    split(-1, 0)
    S.test_direct_vjp_at_tile_and_chunk_edges(n, bc)


@pytest.mark.parametrize("bc", ["open", "periodic"])
def test_gradient_in_several_launches_near_and_on_a_line(split, bc):
    split(-1, 0)
    S.test_direct_vjp_near_and_on_a_segments_line(bc)


@pytest.mark.parametrize("targets", [32, 96])
def test_gradient_in_several_launches_equals_one(split, targets):
    """A launch's targets change only how the sources' partial sums are grouped: 700
    points, 1e-13 of the largest."""
    w = S._ring_pair(700)
    ubar = np.random.default_rng(2).normal(0.0, 0.1, w.x.shape)
    one = S._vjp(w, ubar, "periodic")
    split(-1, targets * 24 * 6)  # 24 bytes a target and block of 128 sources
    assert np.abs(S._vjp(w, ubar, "periodic") - one).max() <= 1e-13 * np.abs(one).max()
