import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")
    config.addinivalue_line("markers", "slow: longer CPU runs")
    config.addinivalue_line("markers", "reference: needs the compiled reference (oracle/_ref, built from its sources)")


def pytest_runtest_setup(item):
    if item.get_closest_marker("reference"):
        from oracle import REF_SO
        if not os.path.exists(REF_SO):
            pytest.skip("the compiled reference (oracle/_ref) is not built")


@pytest.fixture(scope="session")
def golden():
    import numpy as np

    def load(name):
        return np.load(os.path.join(GOLDEN, name), allow_pickle=False)
    return load
