"""The voxeliser's culling against every segment by itself: the field of a branch is the smallest of its segments' fields,
bit for bit (a vessel of one segment drops nothing, and the union with nothing keeps its distance)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cerebrosim_b200 import vessel  # noqa: E402


def field(points, radii, lo, n, dx):
    cap = np.zeros((2, 3))
    pk = vessel.Packed(["a"], points, radii, [0], [len(points)], cap, cap, [0.0, 0.0])
    lo = np.asarray(lo, float)
    return vessel.sdf_device(pk, lo, lo + (np.array(n) - 1.5) * dx, dx)


def assert_smallest_of_segments(points, radii, lo, n, dx):
    whole = field(points, radii, lo, n, dx)
    assert tuple(whole.shape) == tuple(n)
    single = torch.stack([field(points[k:k + 2], radii[k:k + 2], lo, n, dx) for k in range(len(points) - 1)])
    assert torch.equal(whole, single.amin(0))


def near_tie(rng, centre, dx, length, amp):
    """A short segment on one side of a brick's centre and one of `length` on the other, at nearly the same distance from
    the corner between them: the long one is all but dropped, and nearest there."""
    diag = rng.choice([-1.0, 1.0], 3) / np.sqrt(3)
    h = 0.5 * dx * np.sqrt(3 * 49)
    across = [np.cross(diag, rng.normal(size=3)) for _ in range(2)]
    v, w = (x / np.linalg.norm(x) for x in across)
    s, (ra, rb) = rng.uniform(0.3, 1.0), rng.uniform(0.1, 0.3, 2)
    near, far = centre - diag * s, centre + diag * (s + 2 * h - ra + rb + rng.uniform(-amp, amp))
    t = rng.uniform(0.3, 0.7, 2) * length
    return np.array([near - 0.02 * w, near + 0.02 * w, far - v * t[0], far + v * t[1]]), np.array([ra, ra, rb, rb])


@pytest.mark.parametrize("length", [10.0, 1e4, 1e5, 1e6])
def test_long_segments(length):
    rng = np.random.default_rng(int(length))
    for _ in range(250):
        lo = rng.uniform(-0.5, 0.5, 3)
        pts, rad = near_tie(rng, lo + 0.35, 0.1, length, 1e-5 + 1e-7 * length)
        assert_smallest_of_segments(pts, rad, lo, (8, 8, 8), 0.1)


def test_grid_that_begins_far_away():
    """The last brick of a grid of 40,000 voxels: its coordinates are small differences of large numbers."""
    rng = np.random.default_rng(2)
    n = (40000, 8, 8)
    for _ in range(40):
        lo = np.array([-3999.6, 0.2, -0.1]) + rng.uniform(-0.1, 0.1, 3)
        centre = lo + 0.1 * np.array([n[0] - 4.5, 3.5, 3.5])
        pts, rad = near_tie(rng, centre, 0.1, 5.0, 1e-3)
        assert_smallest_of_segments(pts, rad, lo, n, 0.1)


@pytest.mark.parametrize("points", [2, 3, 90, 257, 300])
def test_vessels(points):
    """Branches of one to several chunks of segments, some points twice (segments of length zero) or a hair apart."""
    rng = np.random.default_rng(points)
    t = np.linspace(0, 1, points)
    pts = np.column_stack([4 * t, np.sin(6 * t), np.cos(4 * t)]) + rng.normal(scale=1e-3, size=(points, 3))
    pts[points // 2] = pts[points // 2 - 1]
    pts[-1] = pts[-2] + 3e-7
    assert_smallest_of_segments(pts, rng.uniform(0.2, 0.8, points), [-1.0, -2.0, -2.0], (41, 35, 33), 0.13)
