"""Batches and configurations of a scan put together in one launch.

With the default batch or a larger one, a scan of a small grid puts positions
and configurations together up to 64 MB of waves per launch (at 256^2: 128
waves).  Checked against the same scan with one launch sequence per batch and
configuration (JMS_SetPassFusion(0)), whose waves are the same: the detector
sums agree to the last place of their FP32 results (2^-23) and the binned patterns to
the order of their float atomics.
"""
import numpy as np
import pytest

from tests import golden_cases as G
from tests import product_cases as PC

pytestmark = pytest.mark.gpu
GPU = 2


@pytest.fixture()
def J():
    import jmultislicelib_b200 as jb

    j = jb.JMS()
    yield j
    j.L.JMS_SetScanBatch(32)
    j.L.JMS_SetPassFusion(1)


def _setup(J, n, nobj=5, nvar=3, flags=G.INT):
    a = 0.045 * n
    J.cleanup()
    J.set_high_tension(300.0)
    J.set_grid(n, n, a, a, 0.4)
    pro = J.calc_propagator(0.19525, 0.0, 0.0, 1)
    probe = J.calc_probe(22.0)
    pgr = PC.synthetic_specimen(n, n, 2, nvar, 3 + n)
    assert J.setup(GPU, [nvar, nvar], np.arange(nobj) % 2, [0, 0], 2, 2, flags) == [0, 0, 0, 0]
    for s in range(2):
        assert J.set_phase_grating(GPU, s, pgr[s]) == 0
    assert J.set_propagator(GPU, 0, pro) == 0
    for i, (b0, b1) in enumerate(((0, 10), (20, 50))):
        assert J.set_detector(GPU, i, *J.calc_ring_detector(b0, b1)) == 0
    assert J.init_core(GPU) == 0
    assert J.set_incident_wave(GPU, probe) == 0
    return a


def _launches(J, fuse, pos, npass, **kw):
    J.L.JMS_SetPassFusion(fuse)
    n0 = J.L.JMS_KernelLaunches()
    e, out, ob = J.scan(pos, npass, **kw)
    assert e == 0, e
    return out, ob, J.L.JMS_KernelLaunches() - n0


def _close(a, b, rel):
    assert np.abs(b).max() > 0
    assert np.abs(a.astype(np.float64) - b).max() <= rel * np.abs(b).max()


@pytest.mark.parametrize("batch", [1, 8, 31])
def test_a_smaller_batch_bounds_the_waves_of_a_launch(J, batch):
    """A batch below the default is the caller's bound on the waves in flight: no batches are put together."""
    a = _setup(J, 128)
    pos = np.random.default_rng(2).uniform(0, a, (40, 2)).astype(np.float32)
    J.L.JMS_SetScanBatch(batch)
    varseq = np.zeros((1, 5), np.int32)
    got, _, n1 = _launches(J, 1, pos, 1, varseq=varseq)
    ref, _, n0 = _launches(J, 0, pos, 1, varseq=varseq)
    assert n1 == n0, (n1, n0)
    np.testing.assert_array_equal(got, ref)


def test_channels_of_a_scan(J):
    """A launch of one wave without a binned pattern adds to the context's channels; in a context that keeps any, the
    scan's launches are those of its batches."""
    flags = G.INT | G.DIF | G.IMG
    n, nd = 64, 4
    a = _setup(J, n, flags=flags)
    pos = np.random.default_rng(4).uniform(0, a, (33, 2)).astype(np.float32)    # the last batch holds one position
    varseq = np.random.default_rng(5).integers(0, 3, (2, 5)).astype(np.int32)
    got = []
    for fuse in (1, 0):
        J.seed(3)
        assert J.offset(GPU, 0.1, 0.2) == 0
        assert J.gpu_multislice(0, 0, 1.0) == 0
        assert J.num_det_planes() == nd
        before = J.get_result(GPU, G.DIF, nd * n * n)
        out, _, _ = _launches(J, fuse, pos, 2, varseq=varseq)
        dif, img = J.get_result(GPU, G.DIF, nd * n * n), J.get_result(GPU, G.IMG, nd * n * n)
        assert np.abs(dif - before).max() > 0
        got.append((out, dif, img))
    for x, y in zip(*got):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("npos,npass", [(50, 5), (300, 2), (129, 3)])
def test_uneven_groups(J, npos, npass):
    """At 256^2 (128 waves a launch): configurations in groups of 2, 2, 1; positions in groups of 128, 128, 44 and of
    128, 1, whose results lie past the first group's."""
    a = _setup(J, 256)
    rng = np.random.default_rng(npos)
    pos = rng.uniform(0, a, (npos, 2)).astype(np.float32)
    varseq = rng.integers(0, 3, (npass, 5)).astype(np.int32)
    got, gb, n1 = _launches(J, 1, pos, npass, varseq=varseq, bin=4)
    ref, rb, n0 = _launches(J, 0, pos, npass, varseq=varseq, bin=4)
    assert n1 < n0
    _close(got, ref, 2.0 ** -23)
    _close(gb, rb, 1e-6)


def test_draws_of_merged_batches(J):
    """Without a variant sequence every batch of 32 positions draws its own configurations, in the order of the
    sequential form, and leaves the generator where that form does."""
    a = _setup(J, 256)
    pos = np.random.default_rng(8).uniform(0, a, (50, 2)).astype(np.float32)
    got = []
    for fuse in (1, 0):
        J.seed(21)
        out, _, n = _launches(J, fuse, pos, 3)
        nxt, _, _ = _launches(J, fuse, pos[:1], 1)
        got.append((out, nxt, n))
    assert got[0][2] < got[1][2]
    _close(got[0][0], got[1][0], 2.0 ** -23)
    np.testing.assert_array_equal(got[0][1], got[1][1])
