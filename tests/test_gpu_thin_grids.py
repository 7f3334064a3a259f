"""Launch grids that outgrow their 65535-block y dimension: many small FP64
solves (more than 65535 of the smallest row tiles) and fields of a few columns
and more rows than 65535 marches, against the FP64 oracle."""

import numpy as np
import pytest

import finitevolx_b200 as fvx
from oracle import fvx_oracle as O

pytestmark = pytest.mark.gpu


# 65537 x 16 rows are 65537 tiles of 16; 1 050 000 rows of 7 (FP32 data of this
# size runs the FP64 chain); an odd, ragged number of 32-row fields.  Bars as in
# the other FP64 chain checks: 1e-12, FP32 output 2e-7 (2^-24 of the result's rounding).
@pytest.mark.parametrize("bc", ["dst", "dct"])
@pytest.mark.parametrize("batch,ny,nx,dtype,tol", [(65537, 16, 16, "float64", 1e-12), (150001, 7, 15, "float32", 2e-7),
                                                   (32801, 32, 8, "float64", 1e-12)])
def test_many_small_solves(cuda_ok, bc, batch, ny, nx, dtype, tol):
    import torch
    from finitevolx_b200.solvers.spectral import DSTHelmholtzPlan
    gen = torch.Generator(device="cuda").manual_seed(batch)
    f = torch.randn(batch, ny, nx, device="cuda", dtype=getattr(torch, dtype), generator=gen)
    got = DSTHelmholtzPlan(ny, nx, 0.1, 0.2, (1.5,), batch, bc=bc).solve(f)
    for b in (0, 1, batch // 2, batch - 2, batch - 1):
        ref = O.spectral_solve(f[b].double().cpu().numpy(), 0.1, 0.2, 1.5, bc)
        assert np.abs(got[b].double().cpu().numpy() - ref).max() <= tol * np.abs(ref).max()

# rows above 16 x 65535, and a size whose marches have 8 rows; FP64 1e-13 of the
# largest value, as the other shapes of these operators.
@pytest.mark.parametrize("shape", [(1048577, 3), (600001, 3)])
def test_tall_shallow_water_fields(cuda_ok, shape):
    import torch
    ny, nx = shape
    rng = np.random.default_rng(7)
    u, v, f = (rng.standard_normal(shape) for _ in range(3))
    grid = fvx.ArakawaCGrid2D(Nx=nx, Ny=ny, Lx=0.3 * nx, Ly=0.2 * ny, dx=0.3, dy=0.2)
    t = [torch.tensor(a, device="cuda") for a in (u, v, f)]
    for got, ref in ((fvx.Coriolis2D(grid)(*t), O.coriolis2d(u, v, f)),
                     (fvx.MomentumAdvection2D(grid)(t[0], t[1], "al"), O.momentum_advection(u, v, 0.3, 0.2, "al"))):
        for g, r in zip(got, ref):
            assert np.abs(g.cpu().numpy() - r).max() <= 1e-13 * max(np.abs(r).max(), 1.0)
