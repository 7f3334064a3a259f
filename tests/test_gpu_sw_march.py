"""The shallow-water march (csrc/sw.cu) and the Jacobian's short walk against
the oracle at warp (30 columns), block (120) and march edges; FP64 1e-13 of the
largest value (sums of a handful of terms, quotients as products), FP32 1e-5."""

import numpy as np
import pytest

import finitevolx_b200 as fvx
from oracle import fvx_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 3), (5, 31), (9, 32), (33, 121), (401, 260), (660, 700)])
@pytest.mark.parametrize("masked", [False, True])
def test_shallow_water_shapes(cuda_ok, shape, masked):
    import torch
    ny, nx = shape
    rng = np.random.default_rng(ny + nx)
    u, v, q, f = (rng.standard_normal(shape) for _ in range(4))
    h = 1.0 + 0.2 * rng.random(shape)
    hm = np.kron(rng.random((ny // 5 + 1, nx // 5 + 1)) > 0.25, np.ones((5, 5), bool))[:ny, :nx]
    mask = fvx.Mask2D.from_mask(hm) if masked else None
    om = {k: np.asarray(a, np.float64) for k, a in O.mask2d_from_mask(hm).items()} if masked else None
    grid = fvx.ArakawaCGrid2D(Nx=nx, Ny=ny, Lx=0.3 * nx, Ly=0.2 * ny, dx=0.3, dy=0.2)
    for dtype, tol in ((torch.float64, 1e-13), (torch.float32, 1e-5)):
        t = [torch.tensor(a, dtype=dtype, device="cuda") for a in (u, v, q, f, h)]
        ur, vr, qr, fr, hr = (a.double().cpu().numpy() for a in t)
        vort, mom = fvx.Vorticity2D(grid, mask), fvx.MomentumAdvection2D(grid, mask)
        pairs = [(fvx.Coriolis2D(grid, mask)(t[0], t[1], t[3]), O.coriolis2d(ur, vr, fr, om)),
                 ([vort.potential_vorticity(t[0], t[1], t[4], t[3])],
                  [O.potential_vorticity_x(ur, vr, hr, fr, 0.3, 0.2, om)]),
                 (vort.pv_flux_energy_conserving(t[2], t[0], t[1]), O.pv_flux(qr, ur, vr, "energy", mask=om)),
                 (vort.pv_flux_enstrophy_conserving(t[2], t[0], t[1]), O.pv_flux(qr, ur, vr, "enstrophy", mask=om)),
                 (vort.pv_flux_arakawa_lamb(t[2], t[0], t[1], alpha=0.3), O.pv_flux(qr, ur, vr, "al", 0.3, om))]
        for s in ("energy", "enstrophy", "al"):
            pairs.append((mom(t[0], t[1], s), O.momentum_advection(ur, vr, 0.3, 0.2, s, om)))
        for got, ref in pairs:
            for g, r in zip(got, ref):
                g = g.double().cpu().numpy()
                np.testing.assert_array_equal(np.isnan(g), np.isnan(r))
                g, r = np.nan_to_num(g), np.nan_to_num(r)
                assert np.abs(g - r).max() <= tol * max(np.abs(r).max(), 1.0)


@pytest.mark.parametrize("shape", [(3, 3), (6, 130), (7, 131), (19, 129), (2, 40, 300), (700, 1100)])
def test_jacobian_walks(cuda_ok, shape):
    import torch
    rng = np.random.default_rng(3)
    f, g = rng.standard_normal(shape), rng.standard_normal(shape)
    got = fvx.arakawa_jacobian(torch.tensor(f, device="cuda"), torch.tensor(g, device="cuda"), 0.1, 0.3)
    ref = O.arakawa_jacobian(f, g, 0.1, 0.3)
    assert np.abs(got.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()
