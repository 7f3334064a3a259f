"""Weight gradients of an empty batch are zero."""

import pytest
import torch

from finitevolx_b200._lib import P, fn, stream_ptr

pytestmark = pytest.mark.gpu


def test_empty_batch(cuda_ok):
    cin, cout, h, w = 16, 16, 32, 32
    x = torch.ones(4, device="cuda")
    wt = torch.ones(cout, cin, 3, 3, device="cuda").bfloat16()
    dw, db = torch.ones(cout, cin, 3, 3, device="cuda"), torch.ones(cout, device="cuda")
    part = torch.full((cout * (cin * 9 + 1),), float("nan"), device="cuda")
    assert fn("fvx_nn_conv_bwd")(P(x), 0, 0, cin, P(wt), P(x), P(x), cout, h, w, 0, P(x), P(None), P(x), P(None), P(dw),
                                 P(db), P(part), stream_ptr()) == 0
    assert not dw.any() and not db.any()
