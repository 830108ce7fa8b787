"""Passes over pairs of waves (several waves in one launch).

A scan whose launch has more points than single waves hold in registers at once
runs its waves two to a thread in packed arithmetic; smaller launches and single
runs take one wave a thread.  Both do
the same operations on a wave, so a scan in batches large enough for pairs
equals, bit for bit, the same scan one wave at a time: on square and
non-square grids, at odd wave counts (the last pair repeats its first wave),
with pairs of different configurations (odd position counts, one position),
and with sub-frame gratings.  So do row lines that run under barriers of their
own (rounded up to 16 or 32 threads, or of two warps).  The count of launches
in pairs shows which form ran.  Every candidate plan of the lengths that have
pairs is compared too, and plasmon paths, whose draws depend on the batch, with
the FP64 oracle.
"""
import numpy as np
import pytest

from tests import golden_cases as G
from tests import product_cases as PC

pytestmark = pytest.mark.gpu
GPU = 2
TOL = 1e-4
# lines of more than 16 values a thread: no pairs on grids with such an axis
LONG = {320, 384, 480, 640, 720, 768, 960, 1024, 2048}
RESIDENT = 148 * 1024 * 16      # points from which a launch takes pairs


@pytest.fixture(scope="module")
def J():
    import jmultislicelib_b200 as jb

    return jb.JMS()


def _setup(J, nx, ny, nobj, nvar, npg=None):
    a, b = 0.045 * nx, 0.045 * ny
    J.cleanup()
    wl = J.set_high_tension(300.0)
    J.set_grid(nx, ny, a, b, 0.4)
    pro = J.calc_propagator(0.19525, 0.0, 0.0, 1)
    dets = [J.calc_ring_detector(b0, b1) for (b0, b1) in ((0, 10), (20, 50), (80, 200))]
    probe = J.calc_probe(22.0)
    gx, gy = npg or (nx, ny)
    pgr = PC.synthetic_specimen(gx, gy, 2, nvar, 17)
    objslc = np.arange(nobj) % 2
    assert J.setup(GPU, [nvar, nvar], objslc, [0, 0], 2, 3, G.INT, npg) == [0, 0, 0, 0]
    for s in range(2):
        assert J.set_phase_grating(GPU, s, pgr[s]) == 0
    assert J.set_propagator(GPU, 0, pro) == 0
    for i, (d, m) in enumerate(dets):
        assert J.set_detector(GPU, i, d, m) == 0
    assert J.init_core(GPU) == 0
    assert J.set_incident_wave(GPU, probe) == 0
    return dict(a=a, b=b, wl=wl, pro=pro, dets=dets, probe=probe, pgr=pgr, objslc=objslc)


@pytest.mark.parametrize("nx,ny,npos,npass,npg", [
    (512, 512, 4, 2, None), (512, 512, 5, 1, None), (512, 256, 3, 3, None), (256, 256, 11, 1, None),
    (256, 192, 1, 12, None), (192, 240, 13, 1, None), (128, 128, 19, 3, None), (128, 64, 39, 1, (64, 32)),
    (64, 64, 39, 1, None), (64, 48, 13, 3, None), (16, 16, 300, 1, None), (180, 180, 20, 1, None),
    # a long axis; row lines rounded up to 32 threads, and of two warps: no pairs, but lines that run by themselves
    (320, 160, 9, 1, None), (720, 48, 40, 1, None), (480, 64, 40, 1, None), (384, 48, 40, 1, None),
    (2048, 64, 12, 1, None),
    # a long axis in a launch too large for the other axis's passes to load their operands early
    (1024, 512, 7, 1, None), (512, 1024, 7, 1, None), (768, 256, 13, 1, None), (256, 768, 13, 1, None),
    (640, 192, 20, 1, None), (192, 640, 20, 1, None), (480, 240, 22, 1, None), (240, 480, 22, 1, None),
    (320, 128, 61, 1, None), (128, 320, 61, 1, None), (1024, 64, 38, 1, None), (64, 1024, 38, 1, None),
    # from the fewest waves that take pairs on
    (512, 512, 5, 2, None), (512, 512, 11, 1, None), (512, 256, 7, 3, None), (256, 256, 37, 1, None),
    (256, 192, 1, 51, None), (192, 240, 53, 1, None), (128, 128, 51, 3, None), (128, 64, 297, 1, (64, 32)),
    (64, 64, 593, 1, None), (64, 48, 265, 3, None), (180, 180, 75, 1, None), (16, 16, 9473, 1, None)])
def test_pairs_equal_single_waves(J, nx, ny, npos, npass, npg):
    st = _setup(J, nx, ny, 5, 3, npg)
    rng = np.random.default_rng(nx + ny + npos)
    pos = rng.uniform(0, [st["a"], st["b"]], (npos, 2)).astype(np.float32)
    varseq = rng.integers(0, 3, (npass, 5)).astype(np.int32)
    got = {}
    try:
        for batch in (npos * npass + 1, 1):
            J.L.JMS_SetScanBatch(batch)
            J.L.JMS_SetPassFusion(int(batch > 1))     # 0: batches are not put together
            n0 = J.L.JMS_PairLaunches()
            e, out, ob = J.scan(pos, npass, varseq=varseq, bin=2)
            assert e == 0, e
            assert (J.L.JMS_PairLaunches() > n0) == (
                batch > 1 and not LONG & {nx, ny} and npos * npass * nx * ny >= RESIDENT)
            got[batch == 1] = out, ob
    finally:
        J.L.JMS_SetScanBatch(32)
        J.L.JMS_SetPassFusion(1)
    # the detector sums of a position's configurations are added in FP64 in either form
    assert np.abs(got[0][0] - got[1][0]).max() <= 1e-7 * np.abs(got[1][0]).max()
    if npass == 1:
        np.testing.assert_array_equal(got[0][0], got[1][0])
    assert np.abs(got[0][1] - got[1][1]).max() <= 1e-6 * np.abs(got[1][1]).max()


@pytest.mark.parametrize("n", [64, 128, 256, 512])
def test_every_candidate_plan_in_pairs(J, n):
    """The plans an autotuner may pick: row candidates with the default columns, column candidates with the default
    rows, an odd count of waves that takes pairs."""
    st = _setup(J, n, n, 4, 2)
    npos = -(-RESIDENT // (n * n)) | 1
    pos = np.random.default_rng(n).uniform(0, st["a"], (npos, 2)).astype(np.float32)
    varseq = np.zeros((1, 4), np.int32)
    k = J.L.JMS_PlanCount(n)
    assert k > 1
    try:
        for ir, ic in [(i, 0) for i in range(k)] + [(0, i) for i in range(1, k)]:
            assert J.L.JMS_SelectPlans(ir, ic) == 0
            got = []
            for batch in (npos, 1):
                J.L.JMS_SetScanBatch(batch)
                n0 = J.L.JMS_PairLaunches()
                e, out, ob = J.scan(pos, 1, varseq=varseq, bin=2)
                assert e == 0, e
                assert (J.L.JMS_PairLaunches() > n0) == (batch > 1)
                got.append((out, ob))
            np.testing.assert_array_equal(got[0][0], got[1][0], err_msg=str((ir, ic)))
            assert np.abs(got[0][1] - got[1][1]).max() <= 1e-6 * np.abs(got[1][1]).max()
    finally:
        J.L.JMS_SetScanBatch(32)
        J.L.JMS_SelectPlans(0, 0)


def test_pairs_with_plasmon_paths(J):
    """Each wave of a pair takes its own plasmon path (grid 64^2, 593 waves; some of them, with the last, which has no
    partner, against the oracle)."""
    from oracle import oracle as OR

    c = G.case("msh")
    PC.setup_case(J, c)
    nobj, npos = len(c["objslc"]), 593
    pos = np.random.default_rng(3).uniform(0, c["a"], (npos, 2)).astype(np.float32)
    varseq = OR.Rng(5).variant_sequence(c["nvar"], c["objslc"])[None]
    J.seed(44)
    J.L.JMS_SetScanBatch(npos)
    n0 = J.L.JMS_PairLaunches()
    try:
        e, out, _ = J.scan(pos, 1, varseq=varseq)
        assert J.L.JMS_PairLaunches() > n0
    finally:
        J.L.JMS_SetScanBatch(32)
        J.L.SetPlasmonMC(0, 0.0, 0.0, 0.0, 0)
    assert e == 0
    qe, qc, mfp, nmax = (float(v) for v in c["plasmon"])
    rng = OR.Rng(44)
    n, hsh = OR.detection_planes(c["ndetper"], nobj)
    base = np.concatenate([[0], np.cumsum(c["nvar"])[:-1]]).astype(np.int64)
    for iw in range(npos):
        path = rng.plasmon_shifts(c["slcthick"][c["objslc"]], np.float32(c["a"]), np.float32(c["b"]), qe, qc, mfp,
                                  int(nmax))
        if iw % 37 > 1 and iw + 1 < npos:
            continue
        w0 = OR.offset(c["probe"], c["a"], c["b"], c["wl"], float(pos[iw, 0]), float(pos[iw, 1]))
        ref = OR.multislice(w0, np.concatenate(c["pgr"]), (base[c["objslc"]] + varseq[0]).astype(np.int32),
                            np.stack(c["pro"]), c["proidx"][c["objslc"]], hsh, n, det=np.stack(c["det"]),
                            masks=c["msk"], imagedet=G.INT, weight=1.0, shifts=path)["det_int"][:, :c["ndet"]]
        den = np.maximum(np.abs(ref).max(axis=0), 1e-3)
        assert (np.abs(out[iw] - ref).max(axis=0) / den).max() < TOL
