import gc
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")


@pytest.fixture(scope="session")
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def pytest_runtest_setup(item):
    # the no-allocation checks compare torch's allocated bytes across a call: tensors of
    # earlier tests that are kept only by reference cycles are freed before, not during
    if item.path.name == "test_zz_no_alloc.py":
        gc.collect()
