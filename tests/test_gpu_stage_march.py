"""The fused stage's column march (csrc/march.cuh, csrc/qg_stage.cuh) against
the FP64 oracle where it can go wrong: grids smaller than a tile or a march,
tile remainders in both directions, the first and last rows and columns, every
tile shape and scheme, walls, and the extra terms."""

import numpy as np
import pytest

import finitevolx_b200 as fvx
from oracle import fvx_oracle as O

pytestmark = pytest.mark.gpu


def _check(ny, nx, method, bc, dtype, tol, **kw):
    import torch
    rng = np.random.default_rng(ny * 131 + nx)
    q = np.zeros((ny + 2, nx + 2))
    q[1:-1, 1:-1] = rng.standard_normal((ny, nx)) * 1e-5
    q = O.enforce_periodic(q) if bc == "periodic" else O.pad_interior_constant(q)
    grid = fvx.ArakawaCGrid2D.from_interior(nx, ny, 1e4 * nx, 1.3e4 * ny)
    lam, dt = 1.0 / 4e4 ** 2, 2000.0
    t = torch.tensor(q, dtype=dtype, device="cuda")
    f = None
    if kw.pop("forced", False):
        f = rng.standard_normal(q.shape) * 1e-11
    ref = O.qg_step(t.double().cpu().numpy(), grid.dx, grid.dy, 1.7e-11, lam, dt, method, bc=bc, forcing=f, **kw)
    model = fvx.QGModel(grid, 1.7e-11, lam, method=method, bc=bc, dtype=dtype, forcing=f, **kw)
    got = model.step(t, dt).double().cpu().numpy()
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()


# interior sizes: below one tile, one column / row over a tile edge (16, 32,
# 64, 128), odd pitches.  Bar: the FP64 step's 1e-12.
@pytest.mark.parametrize("size", [(9, 8), (14, 31), (33, 15), (17, 65), (40, 129)])
@pytest.mark.parametrize("method", ["upwind1", "upwind3", "weno3", "weno5", "wenoz5", "weno7", "weno9", "van_leer",
                                    "minmod"])
def test_every_tile_fp64(cuda_ok, method, size):
    import torch
    from finitevolx_b200 import autotune
    try:
        for cfg in range(len(autotune._TILES)):
            autotune.set_stage_tile(method, torch.float64, cfg)
            _check(*size, method, "periodic" if cfg % 2 else "wall", torch.float64, 1e-12)
    finally:
        autotune.set_stage_tile(method, torch.float64, 5)


@pytest.mark.parametrize("bc", ["periodic", "wall"])
def test_extra_terms_and_fp32(cuda_ok, bc):
    import torch
    _check(37, 70, "weno5", bc, torch.float64, 1e-12, forced=True, drag=1e-7, viscosity=50.0)
    _check(40, 72, "weno5", bc, torch.float32, 1e-5)
    _check(72, 200, "wenoz5", bc, torch.float32, 1e-5, forced=True, drag=1e-7, viscosity=50.0)
