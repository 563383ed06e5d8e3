"""FUN1KO's largest cross diffusion (turb3.f:7385) runs over the storage from
cell (1,1,1) to (IMAX,JMAX,KMAX), the ghost cells between the rows and planes
among them: a value that a host left in SEPS there counts, one before the
first or after the last interior cell does not.  Against the oracle."""
import numpy as np
import pytest

from finflo_b200.gpu import GpuSolver
from oracle.oracle import Oracle
from tests.util import interior, make_pair

pytestmark = pytest.mark.gpu


def _fun1(cell, value):
    bg, bc, prm, _ = make_pair(18, 11, 9, turbulence="sst", reynolds=1e6, mach=0.6, h1=1e-3)
    o = Oracle(bc, prm)
    o.start()
    g = GpuSolver(0)
    bid = g.add_block(bg, prm)
    g.upload(bid)
    g.start(bid)
    g.statim(bid)
    g.residu(bid, 1, 1)
    for n, a in g.download(bid).items():
        bc.arrays[n][:] = a
    s = bc.arrays["SEPS"].reshape(bc.kmax + 4, bc.jmax + 4, bc.imax + 4)
    s[cell] = value
    g.upload(bid, ["SEPS"], src=bc.arrays)
    g.residu(bid, 1, 5)
    got = interior(bg, g.download(bid, ["FUN1"])["FUN1"])
    g.close()
    o.turbeq()
    o.residu_sst(5)
    return got, interior(bc, bc.arrays["FUN1"])


@pytest.mark.parametrize("cell,counts", [((4, 5, 1), True), ((4, 1, 6), True), ((5, 12, 19), True), ((2, 3, 19), True),
                                         ((2, 2, 1), False), ((9, 11, 19), False), ((1, 5, 5), False)])   # storage k, j, i
def test_ghost_values_in_the_storage_range_count(gpu_lib, cell, counts):
    plain, _ = _fun1((1, 1, 1), 0.0)
    got, ref = _fun1(cell, 1e18)
    assert np.abs(got - ref).max() <= 1e-11
    assert (np.abs(ref - plain).max() > 1e-3) == counts
