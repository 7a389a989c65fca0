import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200) and the built liblible_b200.so")


@pytest.fixture(autouse=True)
def reference_library(monkeypatch):
    """Where the reference library is not built (its sources are not part of this repository), a test is skipped
    at its first call into it; what it checks before that has passed."""
    from oracle import ref
    if not ref.available():
        monkeypatch.setattr(ref, "lib", lambda: pytest.skip("reference library not built"))


def pytest_collection_modifyitems(config, items):
    if not os.path.exists(os.path.join(ROOT, "oracle", "_ref", "test_dropin")):
        for item in items:
            if item.path.name == "test_gpu_cxx.py":
                item.add_marker(pytest.mark.skip(reason="C++ drop-in check not built (it needs the reference's headers)"))
    try:
        import torch
        has_gpu = torch.cuda.is_available()
    except Exception:
        has_gpu = False
    if has_gpu:
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)
