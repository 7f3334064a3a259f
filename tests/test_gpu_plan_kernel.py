"""The even/odd product kernel is held per plan: choosing or tuning one leaves
the products of other plans, which pick their form by size, to the bit."""

import pytest
import torch

import finitevolx_b200 as fvx
from finitevolx_b200 import autotune
from finitevolx_b200._lib import fn
from finitevolx_b200.solvers.spectral import DSTHelmholtzPlan

pytestmark = pytest.mark.gpu


def test_kernel_is_per_plan(cuda_ok, tmp_path, monkeypatch):
    monkeypatch.setenv("FVX_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    # 160 tiles: the form by size is the tile walk, another order of sums than
    # the 32-element K blocks of kind 2
    f = torch.randn(80, 256, 256, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    a, b = (DSTHelmholtzPlan(256, 256, 0.1, 0.2, (0.05,), batch_max=80, fp64=False) for _ in range(2))
    by_size = a.solve(f).clone()
    b.set_kernel(2)
    other = b.solve(f).clone()
    assert torch.equal(a.solve(f), by_size)
    fn("fvx_dst_kernel_config")(2)
    try:
        assert torch.equal(a.solve(f), other)
        b.set_kernel(0)
        assert torch.equal(b.solve(f), by_size)
    finally:
        fn("fvx_dst_kernel_config")(0)
    grid = fvx.ArakawaCGrid2D.from_interior(256, 256, 5.12e6, 5.12e6)
    model = fvx.QGModel(grid, 1.7e-11, 1.0 / 4e4 ** 2)
    q = 1e-5 * torch.randn(258, 258, device="cuda")
    autotune.tune_dst_kernel(model, q, 1e4)
    assert fn("fvx_dst_kernel_config")(-1) == 0
    assert torch.equal(a.solve(f), by_size)
    assert fn("fvx_dst_plan_kernel")(a.handle, 3) != 0 and fn("fvx_dst_plan_kernel")(a.handle, -2) != 0
