"""Layer/mode transforms of the ensemble on sizes whose cells are not whole
blocks of the kernels' runs: part of one run, a ragged last run, a ragged last
group of four.  Bar: the ensemble's FP32-step 1e-5."""

import pytest
import torch

import finitevolx_b200 as fvx

from test_gpu_ensemble import _member_errors, init_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("members", [[(40, 3), (40, 1)], [(72, 2), (72, 3)], [(104, 1), (48, 2)]])
def test_ragged_runs_match_oracle(cuda_ok, members):
    ens = fvx.QGEnsemble(members)
    qs = init_state(ens)
    ens.step(1)
    torch.cuda.synchronize()
    errs = _member_errors(ens, qs)
    assert max(errs.values()) < 1e-5, errs
