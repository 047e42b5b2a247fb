import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (ROOT, os.path.join(ROOT, "oracle"), os.path.dirname(os.path.abspath(__file__))):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on a B200 with -m gpu)")


# tests against the reference executables, which fail where these are not built
NEED_REFERENCE = ("test_gpu_scale_parity", "test_gpu_styles", "test_oracle_dump")


def pytest_collection_modifyitems(items):
    """Where the reference executables are not built, what needs them runs last:
    a run that stops at its first failure then stops behind everything else."""
    if not os.path.exists(os.path.join(ROOT, "oracle", "_ref", "cac_eamfix")):
        items.sort(key=lambda item: item.module.__name__ in NEED_REFERENCE)


@pytest.fixture(scope="session")
def oracle_mod():
    import oracle
    oracle.lib()          # builds the C restatement on first use
    return oracle


@pytest.fixture(scope="session")
def golden():
    import numpy as np
    cache = {}

    def load(name):
        if name not in cache:
            cache[name] = dict(np.load(os.path.join(ROOT, "tests", "golden", name + ".npz")))
        return cache[name]
    return load
