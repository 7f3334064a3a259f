"""A mask that is not 0 / 1 (the oracle's arithmetic multiplies by it) is
honoured on every grid size and with an initial guess, not only where the whole
cycle runs in one CTA.  Bars as in the other V-cycle checks: FP64 1e-11, FP32
1e-5."""

import numpy as np
import pytest
import torch

from finitevolx_b200.solvers.multigrid import MultigridSolver
from oracle import fvx_oracle as O

pytestmark = pytest.mark.gpu


def _problem(n, seed=0):
    rng = np.random.default_rng(n + seed)
    m = np.ones((n, n))
    m[0] = m[-1] = m[:, 0] = m[:, -1] = 0.0
    m[10:14, 5:9] = 0.5
    m[n // 2:n // 2 + 3, n // 2:] *= 0.25
    c = np.exp(0.3 * rng.standard_normal((n, n)))
    return m, c, rng.standard_normal((n, n)) * m, rng.standard_normal((n, n))


@pytest.mark.parametrize("dtype,bar", [(torch.float64, 1e-11), (torch.float32, 1e-5)])
@pytest.mark.parametrize("n,guess,kw", [(32, True, {}), (128, False, {}), (128, True, {"n_pre": 3, "n_post": 2}),
                                        (256, False, {"n_pre": 0, "n_post": 1})])
def test_fractional_mask(cuda_ok, n, guess, kw, dtype, bar):
    m, c, f, u = _problem(n)
    u = u if guess else np.zeros_like(u)
    args = dict(lambda_=0.1, coeff=c, **kw)
    ref = O.mg_vcycle(O.mg_build(m, 1.3, 0.9, **args), u, f)
    mg = MultigridSolver(m, 1.3, 0.9, dtype=dtype, **args)
    fd, ud = (torch.tensor(a, dtype=dtype, device="cuda") for a in (f, u))
    got = mg.v_cycle(ud if guess else None, fd).double().cpu().numpy()
    assert np.linalg.norm(got - ref) <= bar * np.linalg.norm(ref)


def test_fractional_mask_hybrid_cycle(cuda_ok):
    import ctypes

    from finitevolx_b200._lib import I, P, check, fn, stream_ptr
    m, c, f, _ = _problem(64)
    ref = O.mg_hybrid(O.mg_build(m, 1.3, 0.9, lambda_=0.1, coeff=c), f, 1, 3, 2)
    mg = MultigridSolver(m, 1.3, 0.9, lambda_=0.1, coeff=c)
    fd = torch.tensor(f, device="cuda")
    out = torch.empty_like(fd)
    check(fn("fvx_mg_vcycle_hybrid")(mg.handle, P(fd), P(out), I(1), I(3), I(2), I(0), I(0), ctypes.c_void_p(0),
                                     ctypes.c_void_p(0), stream_ptr()), "hybrid cycle")
    assert np.linalg.norm(out.cpu().numpy() - ref) <= 1e-11 * np.linalg.norm(ref)
