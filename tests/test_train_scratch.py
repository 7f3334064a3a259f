"""Scratch rows of the weight gradients (host logic, no GPU): one per item of the
strip height a layer runs with, never above the channel-independent bound, which
for the 32-channel layers of the network is twice what they need."""

import ctypes

import pytest

from finitevolx_b200._lib import LIB_PATH


@pytest.fixture(scope="module")
def lib():
    if not LIB_PATH.exists():
        from finitevolx_b200.build import build
        build()
    return ctypes.CDLL(str(LIB_PATH))


def test_rows_follow_the_strip(lib):
    rows, bound = lib.fvx_nn_conv_bwd_rows, lib.fvx_nn_conv_bwd_blocks
    for batch in (1, 2, 7, 32, 64):
        for h, w in ((1, 1), (8, 8), (16, 18), (33, 36), (64, 64), (128, 128)):
            for cin in (1, 3, 16, 32):
                for cout in (1, 16, 32):
                    assert 1 <= rows(batch, cin, cout, h, w) <= bound(batch, h, w)
    assert rows(32, 16, 16, 128, 128) == 592       # 2048 items of 16 rows
    assert rows(32, 32, 32, 32, 32) == 256         # 8-row strips: shared memory
    assert rows(2, 16, 16, 16, 16) == 8            # 4-row strips: few items
    assert rows(1, 0, 16, 16, 16) == rows(1, 16, 33, 16, 16) == rows(0, 16, 16, 16, 16) == -1


def test_network_scratch(lib):
    # (channels in and out, divisor of the grid) of the network at 32 x 128^2:
    # the largest is the 32 to 16 layer at the cap of 592 rows
    layers = [(3, 16, 1), (16, 16, 2), (16, 32, 4), (32, 32, 8), (32, 32, 4), (32, 16, 2), (16, 16, 1), (16, 1, 1)]

    def floats(rows):
        return max(rows(ci, co, 128 // d) * co * (9 * ci + 1) for ci, co, d in layers)

    need = floats(lambda ci, co, n: lib.fvx_nn_conv_bwd_rows(32, ci, co, n, n))
    assert need == 592 * 16 * (9 * 32 + 1)
    assert floats(lambda ci, co, n: lib.fvx_nn_conv_bwd_blocks(32, n, n)) == 512 * 32 * (9 * 32 + 1)
