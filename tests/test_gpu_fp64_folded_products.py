"""The FP64 chain's folded products (csrc/dst_f64.cuh) against the FP64 oracle:
odd and even lengths (a middle column, a first periodic column without a
partner), tile edges and remainders, batches that cross tiles, views whose
rows are not 16-byte aligned, and every tile shape."""

import numpy as np
import pytest

from oracle import fvx_oracle as O

pytestmark = pytest.mark.gpu


def _solve(rhs, bc):
    import torch
    from finitevolx_b200.solvers.spectral import get_plan
    b = int(np.prod(rhs.shape[:-2])) if rhs.ndim > 2 else 1
    return get_plan(*rhs.shape[-2:], 0.1, 0.2, (1.5,), b, bc=bc).solve(rhs).double().cpu().numpy()


# 16- and 32-element tile edges (15 .. 33), single cells, odd x even, batches
# whose rows straddle tiles; (8, 300, 301) and (1, 1100, 900) take the larger
# tiles.  Bars: a K-term FP64 sum rounds to ~sqrt(K) 2^-53 of the result's
# size, four products of K <= 1100 stay below 1e-13; FP32 output adds 2^-24.
@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 2, 3), (2, 15, 16), (3, 17, 31), (1, 33, 32), (5, 63, 65),
                                   (8, 300, 301), (1, 1100, 900)])
@pytest.mark.parametrize("bc", ["dst", "dct", "fft"])
def test_folded_products_match_oracle(cuda_ok, bc, shape):
    import torch
    f = np.random.default_rng(3).standard_normal(shape)
    ref = np.stack([O.spectral_solve(x, 0.1, 0.2, 1.5, bc) for x in f])
    got = _solve(torch.tensor(f, device="cuda"), bc)
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
    if shape[1] % 8 or shape[2] % 8:  # FP32 data of these sizes runs the FP64 chain
        f32 = f.astype(np.float32)
        ref = np.stack([O.spectral_solve(x.astype(np.float64), 0.1, 0.2, 1.5, bc) for x in f32])
        got = _solve(torch.tensor(f32, device="cuda"), bc)
        assert np.abs(got - ref).max() <= 2e-7 * np.abs(ref).max()


def test_null_mode_and_interior_view(cuda_ok):
    import ctypes

    import torch
    from finitevolx_b200._lib import D, I, P, check, fn, stream_ptr
    from finitevolx_b200.solvers.spectral import get_plan
    # lambda = 0: the zero eigenvalue of the cosine and periodic problems divides out as 0
    f = np.random.default_rng(4).standard_normal((40, 37))
    f -= f.mean()
    for bc in ("dct", "fft"):
        ref = O.spectral_solve(f, 0.1, 0.2, 0.0, bc)
        got = get_plan(40, 37, 0.1, 0.2, (0.0,), 1, bc=bc).solve(torch.tensor(f, device="cuda")).cpu().numpy()
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
    # interior views of a ghost-ring field, in place: rows at an 8-byte offset and an odd pitch
    q = np.random.default_rng(5).standard_normal((42, 39))
    plan = get_plan(40, 37, 0.1, 0.2, (1.5,), 1)
    t = torch.tensor(q, device="cuda")
    view = t.view(-1)[39 + 1:]
    n, ld = ctypes.c_longlong(40 * 39), ctypes.c_longlong(39)
    check(fn("fvx_dst_solve_f64")(plan.handle, P(view), n, ld, P(view), n, ld, I(1), I(0), D(0.0), I(1), None,
                                  stream_ptr()), "solve")
    ref = q.copy()
    ref[1:-1, 1:-1] = O.solve_helmholtz_dst(q[1:-1, 1:-1], 0.1, 0.2, 1.5)
    got = t.cpu().numpy()
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
    ring = np.ones_like(q, bool)
    ring[1:-1, 1:-1] = False
    np.testing.assert_array_equal(got[ring], q[ring])
