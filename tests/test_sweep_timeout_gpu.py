"""The bounded waits of the warp-wavefront LU-SGS sweep, with the kernel that has
no patience: the CTAs of even tickets give up on their first record, the others
on their first edge words (the upstream CTA needs microseconds to get there).
The kernels end by themselves, the call reports the time-out, and the same
context then sweeps a new state as if nothing had happened."""
import numpy as np
import pytest

from finflo_b200.gpu import FinfloGpuError, GpuSolver
from tests.util import interior, make_pair

pytestmark = pytest.mark.gpu

SST = dict(turbulence="sst", reynolds=1e6, mach=0.6, h1=1e-3)


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("sst", [False, True])
@pytest.mark.parametrize("dims", [(17, 9, 5), (3, 9, 9), (20, 34, 19)])   # 1, 1 and 5 x 3 CTA tiles
def test_time_out_is_reported_and_forgotten(gpu_lib, dims, sst, fp32):
    bg, _, prm, _ = make_pair(*dims, **(SST if sst else {}))
    names = ["DRO", "DM", "DN", "DW", "DE"] + (["DRK", "DEPS"] if sst else [])
    prm.lusgs_fp32 = fp32
    g = GpuSolver(0)
    bid = g.add_block(bg, prm)
    g.upload(bid)
    g.start(bid)
    g.statim(bid)
    g.residu(bid, 1, 1)
    res = g.download(bid, names)

    def increments():
        g.upload(bid, names, src=res)
        g.imps(bid, 1)
        return {n: interior(bg, a) for n, a in g.download(bid, names).items()}

    want = increments()
    for _ in range(2):
        g.sweep_haste(True)
        with pytest.raises(FinfloGpuError, match="timed out"):
            increments()
        g.sweep_haste(False)
        got = increments()
        for n in names:
            assert np.isfinite(got[n]).all()
            np.testing.assert_array_equal(got[n], want[n])
    g.close()


def test_a_captured_cycle_takes_the_switch(gpu_lib):
    bg, _, prm, _ = make_pair(20, 34, 19)
    g = GpuSolver(0)
    bid = g.add_block(bg, prm)
    g.upload(bid)
    g.start(bid)
    g.cycles(2, bid, icycle0=2)
    g.sweep_haste(True)
    with pytest.raises(FinfloGpuError, match="timed out"):
        g.cycles(2, bid, icycle0=4)
    g.sweep_haste(False)
    g.upload(bid)
    g.start(bid)
    assert np.isfinite(g.cycles(2, bid, icycle0=2)).all()
    g.close()


def test_sweeps_queued_right_after_a_time_out(gpu_lib):
    """The edge words (5.8 MB here) hold their marks again before anything that
    is queued after the call which reported the time-out: many sweeps, each
    started as soon as that call returns, all give the increments of the first."""
    bg, _, prm, _ = make_pair(101, 81, 61)
    names = ["DRO", "DM", "DN", "DW", "DE"]
    g = GpuSolver(0)
    bid = g.add_block(bg, prm)
    g.upload(bid)
    g.start(bid)
    g.statim(bid)
    for _ in range(2):   # the second call finds the ghost cells as every later one does
        g.residu(bid, 1, 1)
    g.imps(bid, 1)
    want = g.download(bid, names)
    for _ in range(10):
        g.residu(bid, 1, 1)
        g.sweep_haste(True)
        g.imps(bid, 1)
        g.sweep_haste(False)
        g.residu(bid, 1, 1)   # queued behind the sweep that times out
        with pytest.raises(FinfloGpuError, match="timed out"):
            g.sync()
        g.imps(bid, 1)
        got = g.download(bid, names)
        for n in names:
            np.testing.assert_array_equal(got[n], want[n])
    g.close()
