"""Shared test setup: import paths, the gpu marker, and small helpers."""
import os
import sys

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(REPO, "hsi-detectors-cuda_b200")
for p in (REPO, PKG):
    if p not in sys.path:
        sys.path.insert(0, p)

GOLDEN = os.path.join(REPO, "tests", "golden", "golden.npz")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")


# Tests that fail where the reference's own library (oracle/_ref, compiled from its sources)
# is not built.
NEEDS_REFERENCE = ("test_cpp_threshold.py", "test_gpu_cli_parity.py", "test_gpu_parity_configs.py",
                   "test_lagged_stream_matches_oracle_with_previous_statistics")


def pytest_collection_modifyitems(config, items):
    """Where that library is missing they run last, so that `-x` stops behind all others."""
    import oracle
    if not oracle.ref_available():
        items.sort(key=lambda item: any(name in item.nodeid for name in NEEDS_REFERENCE))


@pytest.fixture(scope="session")
def golden():
    return np.load(GOLDEN, allow_pickle=False)


@pytest.fixture(scope="session")
def orc():
    import oracle
    oracle.fp64_lib()
    return oracle


@pytest.fixture(scope="session")
def hsi():
    """The product binding; GPU tests fail loudly if the library or device is missing."""
    import torch
    import hsi_b200
    if not torch.cuda.is_available():
        pytest.fail("gpu test run without a CUDA device")
    hsi_b200.lib()
    return hsi_b200
