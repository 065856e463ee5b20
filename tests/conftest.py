import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200) and the built native library")


def pytest_collection_modifyitems(config, items):
    # test_gpu_dropin.py runs a program that is built from the reference's
    # sources; where neither it nor a checkout to build it from exists, its
    # failure would say nothing about this package (and end a run under -x).
    from oracle.ref.build_ref import DEFAULT_REFERENCE
    if os.path.exists(os.path.join(ROOT, "oracle", "_ref", "gyref_dropin")) or os.path.isdir(
            os.path.join(DEFAULT_REFERENCE, "Gyunity", "src")):
        return
    absent = pytest.mark.skip(reason="no reference checkout and no program built from one (oracle/_ref/gyref_dropin)")
    for item in items:
        if item.path.name == "test_gpu_dropin.py":
            item.add_marker(absent)


def golden(name):
    return np.load(os.path.join(GOLDEN, name))


@pytest.fixture(scope="session")
def ctx():
    import gyunity_b200 as g
    c = g.Context(0)
    yield c
    c.close()
