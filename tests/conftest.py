import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")


@pytest.fixture(scope="session")
def cuda_ok():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return True


@pytest.fixture(autouse=True)
def _stage_tiles_by_size(request):
    """A GPU test that sets a stage tile for its scheme leaves none behind."""
    yield
    if request.node.get_closest_marker("gpu"):
        import torch
        from finitevolx_b200 import autotune
        from finitevolx_b200._lib import LIB_PATH, SCHEMES
        if LIB_PATH.exists():
            for method in SCHEMES:
                for dtype in (torch.float32, torch.float64):
                    autotune.set_stage_tile(method, dtype, None)
