import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")
    # a reference folder without its sources counts as an absent one
    ref = os.environ.get("XTS_REFERENCE", "/root/reference")
    if not os.path.exists(os.path.join(ref, "xtsrcmaps", "main.cxx")):
        os.environ["XTS_REFERENCE"] = os.path.join(ref, "absent")


@pytest.fixture(scope="session")
def golden():
    import numpy as np

    def load(name):
        return np.load(os.path.join(GOLDEN, name + ".npz"))

    return load
