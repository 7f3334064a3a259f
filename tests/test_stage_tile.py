"""The stage kernel's tile (host logic, no GPU): by the field's size, set for a
scheme and dtype, and by size again."""

import pytest
import torch

from finitevolx_b200 import autotune
from finitevolx_b200._lib import LIB_PATH, SCHEMES, lib


@pytest.fixture(autouse=True, scope="module")
def built():
    if not LIB_PATH.exists():
        from finitevolx_b200.build import build
        build()


def tile(method, dtype, n):
    return autotune._TILES[lib().fvx_qg_tile_for(SCHEMES[method], int(dtype == torch.float64), n, n)]


BY_SIZE = [(256, "16x16"), (706, "16x16"), (708, "32x16"), (1024, "32x16"), (1378, "32x16"), (1379, "64x16"),
           (1870, "64x16"), (1871, "64x32"), (2048, "64x32")]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_set_and_restored(dtype):
    other = torch.float64 if dtype == torch.float32 else torch.float32
    for n, name in BY_SIZE:
        assert tile("weno5", dtype, n) == name
    autotune.set_stage_tile("weno5", dtype, 3)
    assert tile("weno5", dtype, 256) == "64x32"
    assert tile("weno5", other, 256) == tile("weno3", dtype, 256) == "16x16"
    autotune.set_stage_tile("weno5", dtype, None)
    for n, name in BY_SIZE:
        assert tile("weno5", dtype, n) == name


def test_refused():
    count = lib().fvx_qg_tile_config(5, 0, -1)
    assert count == len(autotune._TILES)
    assert lib().fvx_qg_tile_config(5, 0, count) != 0 and lib().fvx_qg_tile_by_size(32, 0) != 0
    assert lib().fvx_qg_tile_for(5, 2, 8, 8) == -1
