import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (GB300, sm_103a) and the built library")
    config.addinivalue_line("markers", "slow: larger CPU cases")


@pytest.fixture(scope="session")
def golden():
    import numpy as np
    return np.load(os.path.join(ROOT, "tests", "golden", "golden.npz"))


@pytest.fixture(autouse=True)
def default_leaf_heights(request):
    """Every GPU test starts with the leaf heights that users get, whatever an earlier
    test in the process has set."""
    if request.node.get_closest_marker("gpu"):
        import torch
        if torch.cuda.is_available():
            import candmc_gb300 as cm
            cm.set_tuning("leaf_rows", 0)
            cm.set_tuning("pipe_leaf_rows", 0)
    yield
