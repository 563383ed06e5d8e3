"""States in which a divisor is zero or a quotient infinite and the result is
still finite, as the reference's arithmetic has it: a cell of zero pressure
(an infinite pressure ratio stops its time step), a cell of zero omega (an
infinite denominator takes the omega increment to zero) and faces whose
sound speed has no bound of its own (DEDPH = 0, limited by the cells').
Against the oracle, with the tolerances of the same stages elsewhere."""
import numpy as np
import pytest

from finflo_b200.gpu import GpuSolver
from oracle.oracle import Oracle
from tests.util import flux_scale, flux_scale_sst, interior, make_pair

pytestmark = pytest.mark.gpu

SST = dict(turbulence="sst", reynolds=1e6, mach=0.6, h1=1e-3)
DIMS = (18, 11, 9)


def _after_residual(sst):
    bg, bc, prm, _ = make_pair(*DIMS, **(SST if sst else {}))
    names = ["DRO", "DM", "DN", "DW", "DE"] + (["DRK", "DEPS"] if sst else [])
    o = Oracle(bc, prm)
    o.start()
    g = GpuSolver(0)
    bid = g.add_block(bg, prm)
    g.upload(bid)
    g.start(bid)
    g.statim(bid)
    g.residu(bid, 1, 1)
    g.sync()
    for n, a in g.download(bid).items():
        bc.arrays[n][:] = a
    return bg, bc, prm, o, g, bid, names


def _increments_match(bg, bc, o, g, bid, names, changed, sst):
    g.upload(bid, changed, src=bc.arrays)
    g.imps(bid, 1)
    got = g.download(bid, names + ["DTL"])
    g.close()
    (o.imps_sst if sst else o.imps)()
    for n in ["DTL"] + names:
        a, ref = interior(bg, got[n]), interior(bc, bc.arrays[n])
        assert np.isfinite(ref).all()
        assert np.abs(a - ref).max() <= 1e-11 * np.abs(ref).max(), n


@pytest.mark.parametrize("sst", [False, True])
def test_zero_pressure_stops_the_time_step(gpu_lib, sst):
    bg, bc, prm, o, g, bid, names = _after_residual(sst)
    interior(bc, bc.arrays["P"])[3, 4, 5] = 0.0
    interior(bc, bc.arrays["P"])[4, 4, 5] = 0.2 * prm.frspre
    _increments_match(bg, bc, o, g, bid, names, ["P"], sst)
    assert interior(bc, bc.arrays["DTL"])[3, 4, 5] == 0.0


def test_zero_omega_takes_no_omega_increment(gpu_lib):
    bg, bc, prm, o, g, bid, names = _after_residual(True)
    interior(bc, bc.arrays["REPS"])[3, 4, 5] = 0.0
    interior(bc, bc.arrays["PTUR"])[3, 4, 5] = 1.0
    _increments_match(bg, bc, o, g, bid, names, ["REPS", "PTUR"], True)


@pytest.mark.parametrize("sst", [False, True])
def test_sound_speed_of_a_face_is_limited_by_its_cells(gpu_lib, sst):
    bg, bc, prm, o, g, bid, names = _after_residual(sst)
    for n, v in (("RO", 1.0), ("DRDP", 1.0), ("DRDH", -1.0)):   # -DRDP / DRDH - 1 / RO = 0 in every cell
        bc.arrays[n][:] = v
    p = bc.arrays["P"]
    p[:] = 1e5 * (1.0 + 1e-6 * np.random.default_rng(0).standard_normal(p.size))   # DEDRH - PHAT / RO^2 near -1
    g.upload(bid, src=bc.arrays)
    g.residu(bid, 1, 5)
    got = g.download(bid, names)
    g.close()
    if sst:
        o.turbeq()
        o.residu_sst(5)
    else:
        o.residu(1, 5)
    S = flux_scale_sst(o, bc) if sst else flux_scale(o, bc)
    for n in names:
        ref, a = interior(bc, bc.arrays[n]), interior(bg, got[n])
        assert np.isfinite(ref).all()
        assert (np.abs(a - ref) <= 1e-12 * np.maximum(np.abs(ref), S[n])).all(), n
