"""The warp-wavefront LU-SGS sweep at the edges of its 8 x 4-line tiles
against the oracle's IMPS: whole and ragged tiles, one tile, one line of
tiles, five and seven equations."""
import numpy as np
import pytest

from finflo_b200.gpu import GpuSolver
from oracle.oracle import Oracle
from tests.util import interior, make_pair

pytestmark = pytest.mark.gpu

SST = dict(turbulence="sst", reynolds=1e6, mach=0.6, h1=1e-3)


def _imps(dims, sst, fp32=0):
    bg, bc, prm, _ = make_pair(*dims, **(SST if sst else {}))
    names = ["DRO", "DM", "DN", "DW", "DE"] + (["DRK", "DEPS"] if sst else [])
    o = Oracle(bc, prm)
    o.start()
    g = GpuSolver(0)
    prm.lusgs_fp32 = fp32
    bid = g.add_block(bg, prm)
    g.upload(bid)
    g.start(bid)
    assert g.lusgs_kind(bid) % 100 == 1
    g.statim(bid)
    g.residu(bid, 1, 1)
    g.sync()
    for n, a in g.download(bid).items():
        bc.arrays[n][:] = a
    res = {n: bc.arrays[n].copy() for n in names}
    (o.imps_sst if sst else o.imps)()
    for _ in range(2):   # the second sweep finds the edge words as the first one left them
        g.upload(bid, names, src=res)
        g.imps(bid, 1)
    g.sync()
    d = g.download(bid, names)
    g.close()
    return [(n, interior(bg, d[n]), interior(bc, bc.arrays[n])) for n in names]


# nodes: cells are one less in each direction
@pytest.mark.parametrize("sst", [False, True])
@pytest.mark.parametrize("dims", [(17, 9, 5), (3, 3, 3), (12, 10, 6), (9, 33, 3), (6, 4, 34), (40, 24, 15)])
def test_increments_match_oracle(gpu_lib, dims, sst):
    for n, got, ref in _imps(dims, sst):
        assert np.isfinite(got).all()
        err = np.abs(got - ref).max() / (np.abs(ref).max() + 1e-300)
        assert err <= 1e-11, (n, err)


@pytest.mark.parametrize("sst", [False, True])
def test_fp32_increments(gpu_lib, sst):
    # FP32 coefficients and sums: about 2^-24 times the conditioning of the
    # diagonal (1e2..1e3 in the thin cells), far below the FP64 increments
    for n, got, ref in _imps((18, 11, 7), sst, fp32=1):
        rel = np.linalg.norm(got - ref) / (np.linalg.norm(ref) + 1e-300)
        assert rel <= 1e-4, (n, rel)
