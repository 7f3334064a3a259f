"""Training convolutions of one layer, forward and backward, against PyTorch in FP64.

The batched kernels pick their block by the number of blocks, the strip height
of the weight gradient by the number of items and the staging by the row length
and the alignment; each is reached below, with rows of whole and of ragged runs
of four.  Tolerances: n-term FP32 sums, n 2^-24 relative to the sum of
magnitudes at worst: 288 terms give 1.7e-5 for outputs and input gradients; the
weight gradients' sums run over the batch's pixels in short per-thread chains
and are held to 1e-4, as the network's are.
"""

import pytest
import torch
import torch.nn.functional as F

from finitevolx_b200._lib import P, fn, lib, stream_ptr

pytestmark = pytest.mark.gpu
DIRECT, POOL, UP = 0, 1, 2

CASES = [  # mode, batch, cin, cout, h, w
    (DIRECT, 2, 3, 16, 32, 32),
    (DIRECT, 2, 16, 1, 33, 36),     # one output channel, aligned runs
    (DIRECT, 3, 5, 1, 17, 35),      # and without
    (DIRECT, 3, 16, 16, 35, 37),    # ragged rows everywhere
    (DIRECT, 40, 16, 16, 40, 52),   # many blocks, 16-row strips
    (DIRECT, 16, 32, 32, 32, 32),   # 8-row strips, four channels a thread
    (POOL, 2, 16, 32, 33, 34),
    (POOL, 2, 32, 32, 16, 16),      # coarse level
    (POOL, 2, 32, 16, 17, 20),
    (POOL, 20, 16, 16, 64, 36),
    (UP, 2, 32, 32, 32, 32),
    (UP, 2, 32, 16, 34, 38),        # even, not a multiple of four
    (UP, 20, 16, 16, 40, 64),
    (UP, 2, 32, 32, 16, 18),
]


def nrel(a, b):
    return ((a.double().cpu() - b).norm() / b.norm()).item()


def source(x, mode):
    if mode == POOL:
        return F.avg_pool2d(x, 2)
    return x if mode == DIRECT else F.interpolate(x, scale_factor=2, mode="nearest")


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("mode,batch,cin,cout,h,w", CASES)
def test_layer_matches_fp64(cuda_ok, mode, batch, cin, cout, h, w, offset):
    gen = torch.Generator().manual_seed(h * w + mode)
    sh, sw = (h, w) if mode == DIRECT else ((2 * h, 2 * w) if mode == POOL else (h // 2, w // 2))

    def make(*shape):
        return torch.randn(*shape, generator=gen)

    def put(t):  # on the device, `offset` values past an aligned address
        buf = torch.empty(t.numel() + 4, device="cuda", dtype=t.dtype)
        v = buf[offset:offset + t.numel()].view(t.shape)
        v.copy_(t)
        return v

    x, wt, bias = make(batch, cin, sh, sw), make(cout, cin, 3, 3).bfloat16(), make(cout)
    skip, dy, dsrc0 = make(batch, cout, h, w), make(batch, cout, h, w), make(batch, cin, sh, sw)
    xr, wr, br = (t.double().requires_grad_() for t in (x, wt.float(), bias))
    y_ref = F.conv2d(source(xr, mode), wr, br, padding=1) + skip.double()
    y_ref.backward(dy.double())

    xd, wd, bd, sd, dyd, dsrc = put(x), wt.cuda(), bias.cuda(), put(skip), put(dy), put(dsrc0)
    y, g = put(torch.zeros(batch, cout, h, w)), put(torch.zeros(batch, cout, h, w))
    dxin, dskip = put(torch.zeros(batch, cin, h, w)), put(torch.zeros(batch, cout, h, w))
    dw, db = torch.empty(cout, cin, 3, 3, device="cuda"), torch.empty(cout, device="cuda")
    part = torch.empty(lib().fvx_nn_conv_bwd_blocks(batch, h, w) * cout * (cin * 9 + 1), device="cuda")
    st = stream_ptr()
    assert fn("fvx_nn_conv_fwd")(P(xd), mode, batch, cin, P(wd), P(bd), P(sd), P(y), cout, h, w, 0, st) == 0
    want_src = cin in (1, 2, 3, 16, 32)
    assert fn("fvx_nn_conv_bwd")(P(xd), mode, batch, cin, P(wd), P(dyd), P(y), cout, h, w, 0, P(g), P(dskip), P(dxin),
                                     P(dsrc if want_src else None), P(dw), P(db), P(part), st) == 0
    assert nrel(y, y_ref.detach()) < 2e-5
    if want_src:
        assert nrel(dsrc, dsrc0.double() + xr.grad) < 2e-5
    assert nrel(dw, wr.grad) < 1e-4 and nrel(db, br.grad) < 1e-4
    assert torch.equal(dskip, g) and torch.equal(g, dyd)
