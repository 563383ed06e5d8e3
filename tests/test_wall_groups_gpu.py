"""The wall-distance searches (every point for few points or points in no
order; boxes of 32 points, of 32 groups, for long ordered lists) against every
cell's distance to every point, to the bit: group and super-group remainders,
points in order and in random order, coincident points, no points, points that
are not numbers."""
import numpy as np
import pytest

from finflo_b200 import case
from finflo_b200.gpu import GpuSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts", [0, 1, 31, 32, 33, 1024, 1025, 2500])
def test_distance_equals_brute_force(gpu_lib, npts):
    blk, prm, _ = case.bump_case(14, 10, 7)
    rng = np.random.default_rng(npts)
    pts = rng.uniform([-1.0, -1.0, -0.5], [4.0, 2.0, 1.0], size=(npts, 3))
    pts[npts // 2:npts // 2 + 3] = pts[:1]
    _compare(blk, prm, pts)


def _compare(blk, prm, pts):
    g = GpuSolver(0)
    bid = g.add_block(blk, prm)
    g.upload(bid)
    g.wall_distance(bid, pts)
    got = g.download(bid, ["DISTW"])["DISTW"]
    g.close()
    best = np.full(blk.ntot, 1.0e8)
    for p in pts:
        dx, dy, dz = blk.arrays["XC"] - p[0], blk.arrays["YC"] - p[1], blk.arrays["ZC"] - p[2]
        best = np.fmin(best, (dx * dx + dy * dy) + dz * dz)
    np.testing.assert_array_equal(got, np.sqrt(best))


@pytest.mark.parametrize("order", ["rows", "random"])
@pytest.mark.parametrize("npts", [4097, 5120, 5121, 8200])
def test_long_lists(gpu_lib, npts, order):
    """More points than every block compares one by one: rows of two walls in
    order take the boxes, the same points shuffled do not."""
    blk, prm, _ = case.bump_case(14, 10, 7)
    rng = np.random.default_rng(npts)
    t = np.arange(npts)
    side = t >= npts // 2
    x, z = -1.0 + 5.0 * (t % 64) / 63.0, -0.5 + 1.5 * ((t % (npts // 2)) // 64) / (npts // 128)
    pts = np.stack([x, np.where(side, 2.0, -1.0) + 0.05 * np.sin(3.0 * x), z], axis=1)
    pts += 1e-3 * rng.standard_normal(pts.shape)
    pts[100:103] = pts[99]
    pts[200], pts[201], pts[202, 1] = np.nan, np.inf, -np.inf
    if order == "random":
        pts = rng.permutation(pts)
    _compare(blk, prm, np.ascontiguousarray(pts))
