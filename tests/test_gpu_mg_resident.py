"""The V-cycle's single-CTA coarse part held in shared memory (csrc/mg.cu)
against the FP64 oracle: levels of one to four rows per thread, columns that do
not divide the threads, odd and no sweeps, and the sizes and masks it leaves to
the global-memory form.  Bars: FP64 1e-11, as the solver's other checks; FP32
1e-5, about a hundred non-amplifying sweeps of 2^-24."""

import numpy as np
import pytest
import torch

from finitevolx_b200.solvers.multigrid import MultigridSolver
from oracle import fvx_oracle as O

pytestmark = pytest.mark.gpu

CASES = [  # ny, nx, options
    (32, 32, {}),                                  # the whole cycle in one CTA
    (128, 128, {}),                                # FP32 enters at 64 x 64: four rows a thread
    (80, 160, {}),                                 # 40 x 80 (four rows), 20 x 40, 10 x 20
    (192, 96, {"n_pre": 3, "n_post": 1}),          # odd sweeps: the result in the other buffer
    (144, 208, {"n_pre": 0, "n_post": 2}),         # 18 x 26 and 9 x 13
    (64, 48, {"n_coarse": 0}),
    (24, 1000, {"n_levels": 2}),                   # coarsest 12 x 500: too large, global memory
    (96, 96, {"n_levels": 2}),                     # coarsest 48 x 48: likewise
    (68, 60, {"n_levels": 3, "n_coarse": 7}),      # coarsest 17 x 15
    (256, 16, {}),                                 # 128 x 8: one row a thread
]


def problem(ny, nx):
    rng = np.random.default_rng(ny * 7 + nx)
    m = np.ones((ny, nx))
    m[0] = m[-1] = m[:, 0] = m[:, -1] = 0.0
    m[ny // 3:ny // 3 + max(2, ny // 8), nx // 4:nx // 2] = 0.0
    c = np.exp(0.3 * rng.standard_normal((ny, nx)))
    return m, c, rng.standard_normal((ny, nx)) * m


@pytest.mark.parametrize("dtype,bar", [(torch.float64, 1e-11), (torch.float32, 1e-5)])
@pytest.mark.parametrize("ny,nx,kw", CASES)
def test_vcycle_matches_oracle(cuda_ok, ny, nx, kw, dtype, bar):
    m, c, f = problem(ny, nx)
    args = dict(lambda_=0.02, coeff=c, **kw)
    ref = O.mg_vcycle(O.mg_build(m, 1.3, 0.9, **args), np.zeros_like(f), f)
    mg = MultigridSolver(m, 1.3, 0.9, dtype=dtype, **args)
    fd = torch.tensor(f, dtype=dtype, device="cuda")
    got = mg.v_cycle(None, fd)
    assert torch.equal(got, mg.v_cycle(None, fd))
    assert np.linalg.norm(got.double().cpu().numpy() - ref) <= bar * np.linalg.norm(ref)


def test_fractional_mask_small_grid(cuda_ok):
    # a mask that is not 0 / 1 keeps the masked arithmetic on a one-CTA grid
    m, c, f = problem(32, 32)
    m[10:14, 5:9] = 0.5
    ref = O.mg_vcycle(O.mg_build(m, 1.0, 1.0, lambda_=0.1), np.zeros_like(f), f)
    got = MultigridSolver(m, 1.0, 1.0, lambda_=0.1).v_cycle(None, torch.tensor(f, device="cuda")).cpu().numpy()
    assert np.linalg.norm(got - ref) <= 1e-11 * np.linalg.norm(ref)


@pytest.mark.parametrize("k", [-600, -360, 360, 600])
def test_fp64_quotients_scale_exactly(cuda_ok, k):
    # the operator is linear, so a right-hand side scaled by a power of two
    # scales every intermediate exactly: quotients formed by multiplication
    # and remainder (exponents within +-400) and plainly divided ones (beyond)
    # have to agree to the last bit
    m, c, f = problem(128, 128)
    mg = MultigridSolver(m, 1.3, 0.9, lambda_=0.02, coeff=c)
    fd = torch.tensor(f, device="cuda")
    scale = 2.0 ** k
    assert torch.equal(mg.v_cycle(None, fd * scale), mg.v_cycle(None, fd) * scale)
    assert torch.equal(mg.apply(fd * scale), mg.apply(fd) * scale)
