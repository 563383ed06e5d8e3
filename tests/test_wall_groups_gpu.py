"""The grouped wall-distance search (boxes of 32 points, of 32 groups) against
every cell's distance to every point, to the bit: group and super-group
remainders, points in random order, coincident points, no points."""
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
    g = GpuSolver(0)
    bid = g.add_block(blk, prm)
    g.upload(bid)
    g.wall_distance(bid, pts)
    got = g.download(bid, ["DISTW"])["DISTW"]
    g.close()
    best = np.full(blk.ntot, 1.0e8)
    for p in pts:
        dx, dy, dz = blk.arrays["XC"] - p[0], blk.arrays["YC"] - p[1], blk.arrays["ZC"] - p[2]
        best = np.minimum(best, (dx * dx + dy * dy) + dz * dz)
    np.testing.assert_array_equal(got, np.sqrt(best))
