"""A model's own stage tile: tuning one model leaves the others alone, and the
tile the field's size picks gives the step of every other tile (FP32 1e-6, FP64
1e-13: only the order of operations at tile edges differs)."""

import pytest
import torch

import finitevolx_b200 as fvx
from finitevolx_b200 import autotune
from finitevolx_b200._lib import SCHEMES, lib

pytestmark = pytest.mark.gpu


def _model(n, dtype):
    grid = fvx.ArakawaCGrid2D.from_interior(n, n, 5.12e6, 5.12e6)
    model = fvx.QGModel(grid, 1.7e-11, 1.0 / 4e4 ** 2, method="weno5", dtype=dtype)
    gen = torch.Generator(device="cuda").manual_seed(n)
    q = 1e-5 * torch.randn(n + 2, n + 2, device="cuda", dtype=dtype, generator=gen)
    return model, q, 0.5 * 5.12e6 / n


def test_tuning_is_per_model(cuda_ok, tmp_path, monkeypatch):
    monkeypatch.setenv("FVX_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    big, q, dt = _model(512, torch.float64)
    small, _, _ = _model(64, torch.float64)
    picked = autotune.tune_qg_stage(big, q, dt)["tile"]
    assert autotune._TILES[big.stage_tile] == picked and small.stage_tile == -1
    assert lib().fvx_qg_tile_for(SCHEMES["weno5"], 1, 66, 66) == 5
    again, _, _ = _model(512, torch.float64)
    autotune.tune_qg_stage(again, q, dt)  # from the file
    assert again.stage_tile == big.stage_tile


# one size of each range of the rule
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-6), (torch.float64, 1e-13)])
@pytest.mark.parametrize("n", [256, 720, 1400, 1880])
def test_tile_by_size(cuda_ok, n, dtype, tol):
    model, q, _ = _model(n, dtype)
    model._dst_from(q)
    outs = []
    for tile in [-1] + list(range(len(autotune._TILES))):
        model.stage_tile = tile
        out = torch.zeros_like(q)
        model._stage(q, None, out, 0.0, 1.0, 1e3, False, True)
        outs.append(out)
    for out in outs[1:]:
        assert (out - outs[0]).abs().max() <= tol * outs[0].abs().max()
    with pytest.raises(RuntimeError):
        model.stage_tile = len(autotune._TILES)
        model._stage(q, None, out, 0.0, 1.0, 1e3, False, True)
