import os
import sys

import pytest
import torch

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box with -m gpu)")


def pytest_collection_modifyitems(config, items):
    if torch.cuda.is_available():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


@pytest.fixture(autouse=True)
def restore_default_dtype():
    # mirrors the reference's tests/conftest.py:53-56
    yield
    torch.set_default_dtype(torch.float32)


@pytest.fixture(autouse=True)
def no_wait_gave_up(request):
    """No kernel of a GPU test may have left by giving up a wait: its outputs would be unfinished."""
    yield
    if "gpu" in request.keywords and torch.cuda.is_available():
        from lit_gpt_b200 import _cabi

        torch.cuda.synchronize()
        _cabi.raise_wait_errors()


@pytest.fixture
def golden():
    import numpy as np

    def load(name):
        return np.load(os.path.join(GOLDEN, name + ".npz"), allow_pickle=False)

    return load
