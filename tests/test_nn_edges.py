"""Surrogate convolutions and pooling at the edges of their tiles.

Channel counts that are not multiples of the kernels' groups (16 output
channels, chunks of 8 input channels, four output channels of the weight
gradient), pixel counts below, at and above one tile, and non-square images
down to 2 x 2, against the FP64 restatement (oracle/nn_oracle.py).  Bounds: an FP32 sum of n products is
within n * 2^-24 of the sum of their magnitudes; the forward result is then
rounded to BF16 (2^-8 of the value).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Ci,H,W,Co,relu", [
    (1, 1, 2, 2, 1, 0), (3, 9, 4, 6, 17, 1), (16, 8, 2, 2, 16, 0), (5, 17, 6, 2, 5, 1), (37, 3, 16, 12, 33, 0),
    (256, 10, 16, 16, 16, 0), (300, 2, 32, 32, 20, 1), (64, 64, 2, 2, 64, 1)])
def test_conv_edges(B, Ci, H, W, Co, relu):
    import torch

    import jmultislicelib_b200 as jb
    from oracle import nn_oracle as N

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

    eps = 2.0 ** -24
    X, Wt, Bs, DY, Y = f(x), f(w), f(bias), f(dy), f(y)
    ref = N.conv_fwd(X, Wt, Bs, relu=bool(relu))
    mag = N.conv_fwd(np.abs(X), np.abs(Wt), np.abs(Bs), relu=False)
    assert np.all(np.abs(Y - ref) <= 2.0 ** -8 * np.abs(ref) + 1.01 * (9 * Ci + 1) * eps * mag + 1e-30)
    rx, rw, rb = N.conv_bwd(X, Wt, Y, DY, relu=bool(relu))
    mx, mw, mb = N.conv_bwd(np.abs(X), np.abs(Wt), Y, np.abs(DY), relu=bool(relu))
    pix = B * (H // 2) * (W // 2)
    assert np.all(np.abs(f(dx) - rx) <= 4 * Co * eps * mx + 1e-30)
    assert np.all(np.abs(f(dw) - rw) <= pix * eps * mw + 1e-30)
    assert np.all(np.abs(f(db) - rb) <= pix * eps * mb + 1e-30)


@pytest.mark.parametrize("B,C,HW,O", [(1, 1, 1, 1), (33, 5, 3, 31), (256, 64, 1, 30), (70, 64, 4, 65)])
def test_pool_linear_edges(B, C, HW, O):
    import torch

    import jmultislicelib_b200 as jb
    from oracle import nn_oracle as N

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

    eps = 2.0 ** -24
    H, WL, BL, D = f(h), f(wl), f(bl), f(dout)
    mag = np.abs(H).mean(axis=(2, 3)) @ np.abs(WL).T + np.abs(BL)
    assert np.all(np.abs(f(out) - N.pool_linear_fwd(H, WL, BL)) <= (C + HW + 2) * eps * mag)
    rh, rw, rb = N.pool_linear_bwd(H, WL, D)
    mh, mw, mb = N.pool_linear_bwd(np.abs(H), np.abs(WL), np.abs(D))
    assert np.all(np.abs(f(dh) - rh) <= (O + 2) * eps * mh)
    assert np.all(np.abs(f(dwl) - rw) <= (B + HW + 2) * eps * mw)
    assert np.all(np.abs(f(dbl) - rb) <= B * eps * mb)


def test_adam_set_equals_single_steps():
    """One launch over several tensors does what one launch per tensor does."""
    import ctypes as C

    import torch

    import jmultislicelib_b200 as jb

    L = jb.lib()
    sizes = (1, 255, 257, 5000)
    g = torch.Generator(device="cuda").manual_seed(1)
    a = [[torch.rand(n, generator=g, device="cuda") for _ in range(4)] for n in sizes]
    b = [[t.clone() for t in ts] for ts in a]
    ca, cb = ([torch.zeros(n, dtype=torch.bfloat16, device="cuda") if n > 255 else None for n in sizes] for _ in range(2))
    for k, n in enumerate(sizes):
        p, gr, m, v = (t.data_ptr() for t in a[k])
        assert L.JMS_NnAdam(p, gr, m, v, ca[k].data_ptr() if n > 255 else None, n, 1e-3, 0.9, 0.999, 1e-8, 3, None) == 0
    arr = C.c_void_p * len(sizes)
    cols = [arr(*[b[k][i].data_ptr() for k in range(len(sizes))]) for i in range(4)]
    copies = arr(*[None if t is None else t.data_ptr() for t in cb])
    assert L.JMS_NnAdamSet(len(sizes), *cols, copies, (C.c_int * len(sizes))(*sizes), 1e-3, 0.9, 0.999, 1e-8, 3, None) == 0
    assert L.JMS_NnAdamSet(33, *cols, copies, (C.c_int * len(sizes))(*sizes), 1e-3, 0.9, 0.999, 1e-8, 3, None) == 2
    torch.cuda.synchronize()
    for s, t in zip([x for ts in a for x in ts] + [x for x in ca if x is not None],
                    [x for ts in b for x in ts] + [x for x in cb if x is not None]):
        assert torch.equal(s, t)
