"""FP32 reconstructions at the ends of the type's range against the FP64 oracle:
weights over a common denominator are products of up to four smoothness terms,
which leave FP32's range (and that of its flushed reciprocal, 2^126) long
before the fields do.  Amplitudes step through the schemes' thresholds.  Bar:
1e-5 of the largest flux, the FP32 bar of these operators; fluxes near the type's
largest value stay finite."""

import numpy as np
import pytest

import finitevolx_b200 as fvx
from oracle import fvx_oracle as O

pytestmark = pytest.mark.gpu

GRID = fvx.ArakawaCGrid2D(Nx=70, Ny=44, Lx=0.3 * 70, Ly=0.2 * 44, dx=0.3, dy=0.2)


def _fields(amplitude):
    rng = np.random.default_rng(11)
    h = (amplitude * rng.standard_normal((44, 70))).astype(np.float32)
    u, v = (rng.standard_normal((44, 70)).astype(np.float32) for _ in range(2))
    return h, u, v


def _close(got, ref):
    assert np.abs(got.double().cpu().numpy() - ref).max() <= 1e-5 * np.abs(ref).max()


def _check(scheme, amplitude, advect):
    import torch
    h, u, v = _fields(amplitude)
    t = [torch.tensor(a, device="cuda") for a in (h, u, v)]
    h, u, v = (a.astype(np.float64) for a in (h, u, v))
    rec = fvx.Reconstruction2D(GRID)
    _close(getattr(rec, scheme + "_x")(t[0], t[1]), O.face_flux_x(h, u, scheme))
    _close(getattr(rec, scheme + "_y")(t[0], t[2]), O.face_flux_y(h, v, scheme))
    if advect:
        _close(fvx.Advection2D(GRID)(*t, method=scheme), O.advection2d(h, u, v, 0.3, 0.2, scheme))


LARGE = [("weno3", 1e9, 8e10), ("wenoz3", 1e9, 8e10), ("weno5", 8e3, 1e6), ("wenoz5", 5e17, 5e19)]


@pytest.mark.parametrize("scheme,lo,hi", LARGE)
def test_large_jumps(cuda_ok, scheme, lo, hi):
    for amplitude in np.geomspace(lo, hi, 14):
        _check(scheme, amplitude, scheme != "wenoz3")


@pytest.mark.parametrize("scheme", ["weno3", "weno5", "wenoz3"])
@pytest.mark.parametrize("amplitude", [1e13, 1e20, 1e30])
def test_beyond_the_products_range(cuda_ok, scheme, amplitude):
    _check(scheme, amplitude, scheme != "wenoz3")


# differences of 1e-10 and below put WENO-Z3's products, 1e-22 and below
# WENO3's, under FP32's smallest normal number; WENO-Z5 uses WENO-Z3 near edges
@pytest.mark.parametrize("scheme,amplitude", [("wenoz3", 1e-10), ("wenoz3", 1e-13), ("wenoz3", 1e-25), ("wenoz5", 1e-13),
                                              ("weno3", 1e-23), ("weno3", 1e-28)])
def test_small_differences(cuda_ok, scheme, amplitude):
    _check(scheme, amplitude, scheme != "wenoz3")


@pytest.mark.parametrize("scheme", ["weno3", "wenoz3", "weno5", "wenoz5"])
def test_constant_field(cuda_ok, scheme):
    import torch
    for value in (0.0, 1e-30, 3e38):
        h = torch.full((44, 70), value, device="cuda")
        one = torch.ones_like(h)
        got = getattr(fvx.Reconstruction2D(GRID), scheme + "_x")(h, one)[1:-1, 1:-1]
        assert torch.equal(got, h[1:-1, 1:-1])
