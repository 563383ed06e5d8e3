"""Ghost cells in one launch each (REFLEC's two passes, REFCOR with MIR) against
the passes one after the other, to the bit.  A mirror patch listed twice keeps
a block off the one-launch route and changes no value."""
import copy

import numpy as np
import pytest

from finflo_b200 import case, grid
from finflo_b200.gpu import GpuSolver

pytestmark = pytest.mark.gpu

NAMES = ["RO", "P", "PDIFF", "TEMP", "U", "V", "W", "C", "E", "VIS", "CH", "DRDP", "DRDH", "RM", "RN", "RW", "EPS2",
         "VIST", "RK", "REPS"]


@pytest.mark.parametrize("turb", [None, "sst"])
@pytest.mark.parametrize("dims", [(3, 3, 3), (17, 9, 9), (41, 24, 12)])
def test_one_launch_equals_pass_by_pass(gpu_lib, dims, turb):
    out, launches = [], []
    for twice in (False, True):
        blk, prm, _ = case.bump_case(*dims, turbulence=turb, noise=1e-2)
        mir = [p for p in blk.patches if p.ityp == grid.BC_MIR]
        assert mir
        if twice:
            blk.patches.append(copy.copy(mir[0]))
        g = GpuSolver(0)
        bid = g.add_block(blk, prm)
        g.upload(bid)
        g.start(bid)
        g.cycles(2, bid, icycle0=1, use_graph=True)
        out.append(g.download(bid, NAMES))
        launches.append(g.cycle_launches(bid))
        g.close()
    assert launches[0] == launches[1] - 2
    for n in NAMES:
        np.testing.assert_array_equal(out[0][n], out[1][n], err_msg=n)
