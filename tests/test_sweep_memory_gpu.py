"""ff_block_params on a full device.  A change of the implicit stage that needs
more memory than there is reports it and leaves the block as it was, without
captured cycles that hold freed buffers; where the old buffers are gone, the
implicit stage is refused until a call succeeds, and then gives what it gave
before."""
import contextlib

import numpy as np
import pytest

from finflo_b200.case import FFParams
from finflo_b200.gpu import FinfloGpuError, GpuSolver
from tests.util import make_pair

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

NAMES = ["DRO", "DM", "DN", "DW", "DE"]


@contextlib.contextmanager
def _full_device(spare=16 << 20):
    """The device's free memory taken up to a few MB more than `spare` (the driver's own needs)."""
    held, n = [], torch.cuda.mem_get_info()[0] - spare
    try:
        while n >= 1 << 21:
            try:
                held.append(torch.empty(n, dtype=torch.uint8, device="cuda"))
                n = torch.cuda.mem_get_info()[0] - spare
            except torch.OutOfMemoryError:
                n //= 2
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


def _solver(ddadi):
    bg, _, prm, _ = make_pair(97, 65, 65)
    prm.ddadi = ddadi
    g = GpuSolver(0)
    bid = g.add_block(bg, prm)
    g.upload(bid)
    g.start(bid)
    g.cycles(2, bid, icycle0=2)
    return g, bid, prm


def test_change_to_lusgs_without_memory(gpu_lib):
    g, bid, prm = _solver(ddadi=1)
    lu = FFParams.from_buffer_copy(prm)
    lu.ddadi = 0
    with _full_device():
        with pytest.raises(FinfloGpuError):
            g.set_params(bid, lu)          # the records take 170 MB
        assert np.isfinite(g.cycles(2, bid, icycle0=4, use_graph=False)).all()
    g.set_params(bid, lu)
    assert np.isfinite(g.cycles(2, bid, icycle0=6)).all()
    g.close()


def test_change_to_ddadi_and_back_needs_no_memory(gpu_lib):
    g, bid, prm = _solver(ddadi=0)
    dd = FFParams.from_buffer_copy(prm)
    dd.ddadi = 1
    for _ in range(2):
        g.residu(bid, 1, 5)
    g.imps(bid, 1)
    want = g.download(bid, NAMES)
    g.set_params(bid, dd)
    g.residu(bid, 1, 5)
    g.imps(bid, 1)
    g.sync()
    with _full_device():
        g.set_params(bid, prm)
        g.residu(bid, 1, 5)
        g.imps(bid, 1)
        got = g.download(bid, NAMES)
    g.close()
    for n in NAMES:
        np.testing.assert_array_equal(got[n], want[n])


def test_change_of_equations_without_memory(gpu_lib):
    g, bid, prm = _solver(ddadi=0)
    for _ in range(2):
        g.residu(bid, 1, 5)
    g.imps(bid, 1)
    want = g.download(bid, NAMES)
    more = FFParams.from_buffer_copy(prm)
    more.iturb = 6                      # seven equations: a fifth more than the old records' memory
    with _full_device():
        with pytest.raises(FinfloGpuError):
            g.set_params(bid, more)
        for call in (lambda: g.imps(bid, 1), lambda: g.cycles(1, bid, icycle0=4), lambda: g.cycles_all(1, icycle0=4),
                     lambda: g.time_stage(4, 1, bid)):
            with pytest.raises(FinfloGpuError, match="no memory"):
                call()
        g.sync()
    g.set_params(bid, prm)
    for _ in range(2):
        g.residu(bid, 1, 5)
    g.imps(bid, 1)
    got = g.download(bid, NAMES)
    for n in NAMES:
        np.testing.assert_array_equal(got[n], want[n])
    g.close()


def test_a_block_takes_the_memory_of_the_setup_scratch(gpu_lib):
    """The set-up calls keep their scratch; a block that needs it gets it."""
    from finflo_b200 import case, grid
    nodes = grid.bump_nodes(97, 65, 65)
    big, _, prm, _ = make_pair(97, 65, 65)
    g = GpuSolver(0)
    bid = g.add_block(big, prm)
    g.block_metrics(bid, *nodes)          # keeps 3 x (nodes + extended nodes) = 21 MB
    small, sprm, _ = case.bump_case(16, 9, 9)
    g.add_block(small, sprm)
    g.sync()
    with _full_device(spare=1 << 20):
        mid, mprm, _ = case.bump_case(25, 17, 17)   # 9 MB of arrays and records
        nid = g.add_block(mid, mprm)
        g.upload(nid)
        g.start(nid)
        assert np.isfinite(g.download(nid, ["RO"])["RO"]).all()
    g.close()
