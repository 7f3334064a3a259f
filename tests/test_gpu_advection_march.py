"""The advection march (csrc/advect.cu) against the FP64 oracle at the places
where it can go wrong: lines shorter than a window, tile and march remainders,
coasts at every distance from the edges, both tile shapes, values whose weight
products overflow, and NaN."""

import numpy as np
import pytest

import finitevolx_b200 as fvx
from oracle import fvx_oracle as O

pytestmark = pytest.mark.gpu
MIN_LEN = {"weno9": 8, "weno7": 6, "weno5": 4, "wenoz5": 4}


def _run(h, u, v, method, mask, dtype):
    import torch
    t = [torch.tensor(a, dtype=dtype, device="cuda") for a in (h, u, v)]
    ny, nx = h.shape
    grid = fvx.ArakawaCGrid2D(Nx=nx, Ny=ny, Lx=0.3 * nx, Ly=0.2 * ny, dx=0.3, dy=0.2)
    adv = fvx.Advection2D(grid, None if mask is None else fvx.Mask2D.from_mask(mask))
    return adv(*t, method=method).double().cpu().numpy(), [a.double().cpu().numpy() for a in t]


def _fields(ny, nx, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((ny, nx)) + 2.0, rng.standard_normal((ny, nx)), rng.standard_normal((ny, nx))


# (1700, 1500) takes the 64 x 32 tiles; the others 32 x 16.  Bars: FP64 1e-12,
# FP32 1e-5 of the largest tendency (the stencils' bars).
@pytest.mark.parametrize("shape", [(4, 3), (8, 9), (17, 33), (31, 65), (70, 40), (1700, 1500)])
@pytest.mark.parametrize("method", O.ADVECTION_METHODS)
def test_sizes_and_masks(cuda_ok, method, shape):
    import torch
    ny, nx = shape
    if min(shape) < MIN_LEN.get(method, 3):
        pytest.skip("shorter than the scheme's ladder")
    if ny > 1000 and method not in ("weno5", "weno9", "van_leer"):
        pytest.skip("one scheme of each reach at the large size")
    h, u, v = _fields(ny, nx, 11)
    rng = np.random.default_rng(12)
    mask = np.kron(rng.random((ny // 7 + 1, nx // 7 + 1)) > 0.25, np.ones((7, 7), bool))[:ny, :nx]
    for m in (None, mask):
        mo = None if m is None else O.mask2d_from_mask(m)
        for dtype, tol in ((torch.float64, 1e-12), (torch.float32, 1e-5)):
            got, (hr, ur, vr) = _run(h, u, v, method, m, dtype)
            ref = O.advection2d(hr, ur, vr, 0.3, 0.2, method, mo)
            assert np.abs(got - ref).max() <= tol * max(np.abs(ref).max(), 1e-300)


@pytest.mark.parametrize("method", ["weno3", "weno5", "wenoz5", "weno7", "weno9", "van_leer"])
def test_overflowing_weights_and_nan(cuda_ok, method):
    # jumps of 1e60 (FP64: the product of two or more squared smoothness
    # measures overflows) keep the form with a division per weight
    import torch
    h, u, v = _fields(40, 70, 13)
    big = h * 1e60
    with np.errstate(over="ignore", invalid="ignore"):
        ref = O.advection2d(big, u, v, 0.3, 0.2, method)
    got, _ = _run(big, u, v, method, None, torch.float64)
    np.testing.assert_array_equal(np.isfinite(got), np.isfinite(ref))
    ok = np.isfinite(ref)
    assert np.abs(got[ok] - ref[ok]).max() <= 1e-11 * np.abs(ref[ok]).max()
    # a NaN and an infinite cell spoil the tendencies the reference's stencils spoil
    h[20, 33] = np.nan
    h[9, 50] = np.inf
    with np.errstate(over="ignore", invalid="ignore"):
        ref = O.advection2d(h, u, v, 0.3, 0.2, method)
    got, _ = _run(h, u, v, method, None, torch.float64)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    ok = np.isfinite(ref)
    np.testing.assert_array_equal(np.isfinite(got), ok)
    assert np.abs(got[ok] - ref[ok]).max() <= 1e-12 * np.abs(ref[ok]).max()
