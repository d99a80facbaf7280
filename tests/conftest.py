import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TESTS = os.path.dirname(os.path.abspath(__file__))
for p in (ROOT, TESTS):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200); parity tests of the CUDA path")


def pytest_collection_modifyitems(items):
    # The reference's own test file runs last: its binary is built from the
    # reference's sources, and where that is absent the failure would end a run
    # that stops at the first one (-x) before the rest of the suite.
    items.sort(key=lambda item: item.path.name == "test_gpu_reference_suite.py")
