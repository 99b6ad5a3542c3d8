import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (ROOT, os.path.join(ROOT, "tests", "golden")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); run with -m gpu")


# The tests that run the reference's own sources, compiled (oracle/_ref, `make -C oracle
# ref dropin`): they need the reference tree, which is not part of this repository
REFERENCE_TESTS = {"test_gpu_dropin.py": None, "test_gpu_prn.py": ("test_shim_section_matches_saver",)}
REFERENCE_BUILDS = ("ref32", "dropin32", "dropin32m", "dropin32r")


def pytest_collection_modifyitems(config, items):
    # GPU tests fail loudly when CUDA is missing instead of silently skipping,
    # unless they were deselected with -m "not gpu".  Only a missing compiled
    # reference skips, and only the tests that run it.
    missing = [k for k in REFERENCE_BUILDS if not os.path.exists(os.path.join(ROOT, "oracle", "_ref", k))]
    if not missing:
        return
    for item in items:
        names = REFERENCE_TESTS.get(os.path.basename(str(item.fspath)), ())
        if names is None or item.name.split("[")[0] in names:
            item.add_marker(pytest.mark.skip(reason="compiled reference not built: oracle/_ref lacks " + ", ".join(missing)))


@pytest.fixture(scope="session")
def cuda_available():
    import torch
    return torch.cuda.is_available()
