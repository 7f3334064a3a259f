"""The FP32 chain's folded tensor-core products (csrc/dst_fold.cuh) against the
FP64 oracle: half lengths below and off the 8-element and 64-element blocks,
row tiles that straddle batches, and each table-row tile (32, 64, 128)."""

import numpy as np
import pytest

from oracle import fvx_oracle as O

pytestmark = pytest.mark.gpu

# (1200, 1000) takes 64-row tiles, 8 x 640^2 128-row ones, the rest 32.  Bar:
# operands carried as bf16 hi + lo (2^-17 relative each) through four
# products, the chain's 1e-4 (about 1e-5 in the 2-norm).
SHAPES = [(1, 8, 8), (2, 16, 24), (3, 120, 136), (1, 256, 512), (1, 1200, 1000), (8, 640, 640)]


def _data(shape, bc):
    f = np.stack([O.kminus3_field(shape[1], shape[2], 7 + k) for k in range(shape[0])]).astype(np.float32)
    lam = 60.0 / (0.1 * shape[2]) ** 2
    ref = np.stack([O.spectral_solve(x.astype(np.float64), 0.1, 0.2, lam, bc) for x in f])
    return f, lam, ref


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bc", ["dst", "dct", "fft"])
def test_folded_split_products_match_oracle(cuda_ok, bc, shape):
    import torch
    from finitevolx_b200.solvers.spectral import DSTHelmholtzPlan
    f, lam, ref = _data(shape, bc)
    plan = DSTHelmholtzPlan(shape[1], shape[2], 0.1, 0.2, (lam,), batch_max=shape[0], bc=bc, fp64=False)
    got = plan.solve(torch.tensor(f, device="cuda")).cpu().numpy()
    plan.check_device()
    assert np.abs(got - ref).max() <= 1e-4 * np.abs(ref).max()
    assert np.linalg.norm(got - ref) <= 2e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("bc", ["dst", "dct", "fft"])
def test_presplit_natural_workspace(cuda_ok, bc):
    # an operand the caller wrote split into the public workspace in natural
    # order (layout 0) gives what the plan makes of the same field
    import ctypes

    import torch
    from finitevolx_b200._lib import I, P, check, fn, stream_ptr
    from finitevolx_b200.solvers.spectral import DSTHelmholtzPlan
    shape = (2, 24, 136)
    f, lam, ref = _data(shape, bc)
    plan = DSTHelmholtzPlan(24, 136, 0.1, 0.2, (lam,), batch_max=2, bc=bc, fp64=False)
    assert fn("fvx_dst_operand_layout")(plan.handle) == 0
    ph, pl = ctypes.c_void_p(), ctypes.c_void_p()
    check(fn("fvx_dst_workspace")(plan.handle, ctypes.byref(ph), ctypes.byref(pl)), "workspace")
    t = torch.tensor(f, device="cuda")
    hi = t.bfloat16()
    lo = (t - hi.float()).bfloat16()
    rt = ctypes.CDLL("libcudart.so.12")  # a plain device-to-device copy into the workspace
    torch.cuda.synchronize()
    for dst, src in ((ph, hi), (pl, lo)):
        assert rt.cudaMemcpy(dst, P(src), ctypes.c_size_t(src.numel() * 2), ctypes.c_int(3)) == 0
    out = torch.empty_like(t)
    check(fn("fvx_dst_solve_presplit_f32")(plan.handle, P(out), ctypes.c_longlong(24 * 136), ctypes.c_longlong(136),
                                           I(2), stream_ptr()), "solve")
    plan.check_device()
    assert np.linalg.norm(out.cpu().numpy() - ref) <= 2e-5 * np.linalg.norm(ref)
