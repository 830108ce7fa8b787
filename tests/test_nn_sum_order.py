"""Order of the surrogate kernels' FP32 sums.

Adam divides a gradient by its own magnitude: within a few training steps
another rounding of a gradient near zero becomes 1e-4 of a bias.  The order of
every sum is therefore part of what the kernels compute, whatever their tiles,
chunks and grids are, and their results equal, bit for bit, a restatement that
rounds to FP32 after each product and addition.  Channel counts off the
kernels' groups, more output channels than one chunk, and pixel and image
counts below and above the 256 threads and images that a sum is dealt to.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CONVS = [
    (1, 1, 2, 2, 1, 0), (3, 9, 4, 6, 17, 1), (16, 8, 2, 2, 16, 0), (5, 17, 6, 2, 5, 1), (37, 3, 16, 12, 33, 0),
    (256, 10, 16, 16, 16, 0), (300, 2, 32, 32, 20, 1), (64, 64, 2, 2, 64, 1), (7, 5, 6, 4, 70, 1)]
POOLS = [(1, 1, 1, 1), (33, 5, 3, 31), (256, 64, 1, 30), (70, 64, 4, 65), (300, 16, 2, 17)]


def _run_conv(B, Ci, H, W, Co, relu):
    """Inputs and results of the three convolution kernels, as float64 arrays."""
    import torch

    import jmultislicelib_b200 as jb

    L = jb.lib()
    rng = np.random.default_rng(B + Ci + H + Co)

    def dev(a, dt):
        return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda().to(dt)

    x = dev(rng.normal(size=(B, Ci, H, W)), torch.bfloat16)
    w = dev(rng.normal(size=(Co, Ci, 3, 3)) / np.sqrt(9 * Ci), torch.bfloat16)
    bias = dev(rng.normal(size=Co), torch.float32)
    dy = dev(rng.normal(size=(B, Co, H // 2, W // 2)), torch.float32)
    y = torch.zeros((B, Co, H // 2, W // 2), dtype=torch.bfloat16, device="cuda")
    dx, dw, db = (torch.full(s, 7.0, device="cuda") for s in ((B, Ci, H, W), (Co, Ci, 3, 3), (Co,)))
    assert L.JMS_NnConvForward(x.data_ptr(), w.data_ptr(), bias.data_ptr(), y.data_ptr(), B, Ci, H, W, Co, relu,
                               None) == 0
    assert L.JMS_NnConvBackward(x.data_ptr(), w.data_ptr(), y.data_ptr(), dy.data_ptr(), dx.data_ptr(), dw.data_ptr(),
                                db.data_ptr(), B, Ci, H, W, Co, relu, None) == 0
    torch.cuda.synchronize()

    def f(t):
        return t.float().cpu().numpy().astype(np.float64)

    return [f(t) for t in (x, w, bias, dy, y, dx, dw, db)]


def _fma(a, b, c):
    """fl32(a b + c): the product is exact in 64-bit mantissas, and a second rounding there moves the result only
    where the sum lies within 2^-40 of a tie of its FP32 spacing."""
    return (np.asarray(a, np.longdouble) * b + c).astype(np.float32)


def _taps(X):
    """[Ci, 3, 3, pixels]: the taps of every output pixel, zero outside the image."""
    B, Ci, H, W = X.shape
    xp = np.zeros((B, Ci, H + 2, W + 2), np.float32)
    xp[:, :, 1:H + 1, 1:W + 1] = X
    t = np.stack([[xp[:, :, ky:ky + H:2, kx:kx + W:2] for kx in range(3)] for ky in range(3)])
    return t.transpose(3, 0, 1, 2, 4, 5).reshape(Ci, 3, 3, -1)


@pytest.mark.parametrize("B,Ci,H,W,Co,relu", CONVS)
def test_conv_sum_order(B, Ci, H, W, Co, relu):
    """Forward: bias, input channel, tap.  Data gradient: tap, output channel.  Weight gradient: the pixels t,
    t + 256, ... of 256 threads, the lanes of a warp in halves (16, 8, 4, 2, 1), the warps."""
    from oracle import nn_oracle as N

    X, Wt, Bs, DY, Y, dx, dw, db = _run_conv(B, Ci, H, W, Co, relu)
    ho, wo = H // 2, W // 2
    taps = _taps(X)
    y = np.repeat(Bs.astype(np.float32)[:, None], B * ho * wo, 1)
    for ci in range(Ci):
        for k in range(9):
            y = _fma(Wt[:, ci, k // 3, k % 3][:, None], taps[ci, k // 3, k % 3], y)
    y = N.bf16_round(np.maximum(y, 0) if relu else y).reshape(Co, B, ho, wo).transpose(1, 0, 2, 3)
    np.testing.assert_array_equal(Y, y)
    g = np.where(Y > 0, DY, 0.0) if relu else DY
    gx = np.zeros((B, Co, ho + 1, wo + 1))             # one more row and column of zeros
    gx[:, :, :ho, :wo] = g
    acc = np.zeros((B, Ci, H, W), np.float32)
    for ky in range(3):
        for kx in range(3):
            py, px = (ky + 1) % 2, (kx + 1) % 2        # parity of the input pixels that see this tap
            at = gx[:, :, (ky == 0):(ky == 0) + ho, (kx == 0):(kx == 0) + wo]
            for co in range(Co):
                acc[:, :, py::2, px::2] = _fma(at[:, co, None], Wt[co, :, ky, kx][:, None, None], acc[:, :, py::2, px::2])
    np.testing.assert_array_equal(dx, acc)

    n = B * ho * wo
    pad = -(-n // 256) * 256
    gp = np.zeros((Co, pad), np.float32)
    gp[:, :n] = g.transpose(1, 0, 2, 3).reshape(Co, n)
    tp = np.ones((10, Ci, pad), np.float32)            # nine taps, and a one for the bias
    tp[:9] = 0
    tp[:9, :, :n] = taps.reshape(Ci, 9, n).transpose(1, 0, 2)
    s = np.zeros((Co, 10, Ci, 256), np.float32)
    for i in range(0, pad, 256):
        s = _fma(gp[:, None, None, i:i + 256], tp[None, :, :, i:i + 256], s)
    s = s.reshape(Co, 10, Ci, 8, 32)
    for h in (16, 8, 4, 2, 1):
        s = s[..., :h] + s[..., h:2 * h]
    t = np.zeros((Co, 10, Ci), np.float32)
    for q in range(8):
        t = t + s[..., q, 0]
    np.testing.assert_array_equal(dw.reshape(Co, Ci, 9), t[:, :9].transpose(0, 2, 1))
    np.testing.assert_array_equal(db, t[:, 9, 0])


def _run_pool(B, C, HW, O):
    import torch

    import jmultislicelib_b200 as jb

    L = jb.lib()
    rng = np.random.default_rng(B + C + O)
    h = torch.from_numpy(rng.normal(size=(B, C, HW, 1)).astype(np.float32)).cuda().to(torch.bfloat16)
    wl, bl, dout = (torch.from_numpy(rng.normal(size=s).astype(np.float32)).cuda() for s in ((O, C), (O,), (B, O)))
    out, dh, dwl, dbl = (torch.zeros(s, device="cuda") for s in ((B, O), (B, C, HW, 1), (O, C), (O,)))
    assert L.JMS_NnPoolLinearForward(h.data_ptr(), wl.data_ptr(), bl.data_ptr(), out.data_ptr(), B, C, HW, O, None) == 0
    assert L.JMS_NnPoolLinearBackward(h.data_ptr(), wl.data_ptr(), dout.data_ptr(), dh.data_ptr(), dwl.data_ptr(),
                                      dbl.data_ptr(), B, C, HW, O, None) == 0
    torch.cuda.synchronize()

    def f(t):
        return t.float().cpu().numpy().astype(np.float64)

    return [f(t) for t in (h, wl, bl, dout, out, dh, dwl, dbl)]


@pytest.mark.parametrize("B,C,HW,O", POOLS)
def test_pool_linear_sum_order(B, C, HW, O):
    """Forward: bias, channel.  Weight gradient: image after image.  Data gradient: output after output."""
    H, WL, BL, D, out, dh, dwl, dbl = _run_pool(B, C, HW, O)
    pooled = np.zeros((B, C), np.float32)
    for k in range(HW):
        pooled = pooled + H.reshape(B, C, HW)[..., k].astype(np.float32)
    pooled = pooled / np.float32(HW)
    s = np.repeat(BL.astype(np.float32)[None], B, 0)
    for c in range(C):
        s = _fma(WL[:, c], pooled[:, c, None], s)
    np.testing.assert_array_equal(out, s)
    w, b = np.zeros((O, C), np.float32), np.zeros(O, np.float32)
    for k in range(B):
        w = _fma(D[k][:, None], pooled[k], w)
        b = b + D[k].astype(np.float32)
    np.testing.assert_array_equal(dwl, w)
    np.testing.assert_array_equal(dbl, b)
    s = np.zeros((B, C), np.float32)
    for o in range(O):
        s = _fma(D[:, o, None], WL[o], s)
    np.testing.assert_array_equal(dh, np.repeat((s / np.float32(HW))[..., None, None], HW, 2))
