"""Batched FP32 even/odd products with more tiles than SMs (one CTA walks
several tiles, csrc/dst.cu) against the FP64 oracle: one tile per CTA and a
few CTAs with two, several tiles per CTA with a ragged last round, a lambda
per batch member, in-place views, and a stalled producer."""

import numpy as np
import pytest

from oracle import fvx_oracle as O

pytestmark = pytest.mark.gpu

# tiles of 128 rows x 2 x 128 columns: 160, 156, 160 and 480 in both directions.
# Bar: operands carried as bf16 hi + lo (2^-17 relative each) through four
# products, the chain's 1e-4 (about 1e-5 in the 2-norm).
SHAPES = [(80, 256, 256), (13, 512, 768), (5, 1024, 1024), (60, 512, 512)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("layers", [1, 2])
def test_tile_walk_matches_oracle(cuda_ok, shape, layers):
    import torch
    from finitevolx_b200._lib import I, fn
    from finitevolx_b200.solvers.spectral import DSTHelmholtzPlan
    B, ny, nx = shape
    if B % layers:
        pytest.skip("members are whole sets of layers")
    base = np.stack([O.kminus3_field(ny, nx, 7 + k) for k in range(3)]).astype(np.float32)
    f = np.stack([base[k % 3] * np.float32(1 + k) for k in range(B)])
    lams = tuple((40.0 + 25.0 * j) / (0.1 * nx) ** 2 for j in range(layers))
    plan = DSTHelmholtzPlan(ny, nx, 0.1, 0.2, lams, batch_max=B, fp64=False)
    t = torch.tensor(f, device="cuda")
    got = plan.solve(t).cpu().numpy()
    plan.check_device()
    refs = {}
    for k in range(B):
        key = (k % 3, k % layers)
        if key not in refs:
            refs[key] = O.spectral_solve(base[key[0]].astype(np.float64), 0.1, 0.2, lams[key[1]], "dst")
        ref = refs[key] * (1 + k)
        assert np.abs(got[k] - ref).max() <= 1e-4 * np.abs(ref).max(), k
        assert np.linalg.norm(got[k] - ref) <= 2e-5 * np.linalg.norm(ref), k
    # the kernel of one tile per CTA, with its own order of the blocks: both
    # carry the same operands, so they agree to FP32 sums of N terms
    fn("fvx_dst_kernel_config")(I(2))
    try:
        other = plan.solve(t).cpu().numpy()
    finally:
        fn("fvx_dst_kernel_config")(I(0))
    assert np.linalg.norm(got - other) <= 2e-5 * np.linalg.norm(other)


def test_stalled_walk_reports_and_recovers(cuda_ok):
    import torch
    from finitevolx_b200._lib import FvxError, fn
    from finitevolx_b200.solvers.spectral import DSTHelmholtzPlan
    plan = DSTHelmholtzPlan(256, 256, 0.1, 0.2, (0.05,), batch_max=80, fp64=False)
    f = torch.tensor(O.kminus3_field(256, 256, 3).astype(np.float32), device="cuda").expand(80, -1, -1).contiguous()
    want = plan.solve(f).clone()
    plan.check_device()
    plan.set_wait_limit(2_000_000)  # ~1 ms
    fn("fvx_dst_plan_inject_stall")(plan.handle, 1)
    try:
        plan.solve(f)
        with pytest.raises(FvxError):
            plan.check_device()
    finally:
        fn("fvx_dst_plan_inject_stall")(plan.handle, 0)
    got = plan.solve(f)
    plan.check_device()
    assert torch.equal(got, want)
