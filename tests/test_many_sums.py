"""A launch with more detector sums than 2^27.

The reduction gives each sum a warp, so its thread count passes 2^32 there:
42,138 positions on 16^2 with 401 planes of 8 detectors.  Positions at both ends
equal, bit for bit, the same positions in a scan of their own.
"""
import ctypes as C

import numpy as np
import pytest

from tests import golden_cases as G
from tests import product_cases as PC

pytestmark = pytest.mark.gpu
GPU = 2


def test_more_than_2_27_sums():
    import torch

    import jmultislicelib_b200 as jb

    J = jb.JMS()
    n, nobj, ndet = 16, 400, 8
    a = 0.045 * n
    J.cleanup()
    J.set_high_tension(300.0)
    J.set_grid(n, n, a, a, 0.4)
    pro, probe = J.calc_propagator(0.19525, 0.0, 0.0, 1), J.calc_probe(22.0)
    pgr = PC.synthetic_specimen(n, n, 2, 1, 5)
    assert J.setup(GPU, [1, 1], np.arange(nobj) % 2, [0, 0], 1, ndet, G.INT) == [0, 0, 0, 0]
    for s in range(2):
        assert J.set_phase_grating(GPU, s, pgr[s]) == 0
    assert J.set_propagator(GPU, 0, pro) == 0
    for i in range(ndet):
        assert J.set_detector(GPU, i, *J.calc_ring_detector(5.0 * i, 5.0 * i + 30.0)) == 0
    assert J.init_core(GPU) == 0
    assert J.set_incident_wave(GPU, probe) == 0
    m = J.num_det_planes() * ndet
    npos = (1 << 27) // m + 300
    pos = np.random.default_rng(6).uniform(0, a, (npos, 2)).astype(np.float32)
    varseq = np.zeros((1, nobj), np.int32)

    def scan(p):
        d_pos = torch.from_numpy(p).cuda()
        out = torch.zeros((len(p), m), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        J.L.JMS_SetScanBatch(len(p))
        assert J.L.JMS_ScanGPUDevice(len(p), d_pos.data_ptr(), 0.0, 1, varseq.ctypes.data_as(C.POINTER(C.c_int)),
                                     out.data_ptr(), None, 0) == 0
        torch.cuda.synchronize()
        return out

    try:
        out = scan(pos)
        assert npos * m > 1 << 27
        for k in (slice(0, 301), slice(npos - 301, npos)):
            ref = scan(pos[k])
            assert ref.abs().max() > 0
            assert torch.equal(out[k], ref)
    finally:
        J.L.JMS_SetScanBatch(32)
        J.cleanup()        # the launch's waves and partial sums, 1.2 GB
