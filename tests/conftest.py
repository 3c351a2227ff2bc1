import os
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (sm_100a B200); run with -m gpu")


# What compares with Alien's own templates (oracle/_ref) needs the reference's headers
# to have been there when the oracle was built: such a test is skipped where they were
# not, from the point on at which it asks for them, or as a whole where it asks in a
# process of its own.
_ASKS_IN_A_PROCESS = {"test_reference_arm_prints_one_complete_json_line"}


def pytest_collection_modifyitems(items):
    from oracle import oracle

    if not oracle.ref_available():
        for item in items:
            if item.name in _ASKS_IN_A_PROCESS:
                item.add_marker(pytest.mark.skip(reason="oracle/_ref not built"))


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    from oracle import oracle

    try:
        return (yield)
    except oracle.ReferenceNotBuilt as e:
        pytest.skip(str(e))


@pytest.fixture(scope="session")
def ctx():
    """One libab2 context on cuda:0 for the GPU tests."""
    from alien_b200 import abi

    c = abi.Context(int(os.environ.get("AB2_DEVICE", "0")))
    yield c
    c.close()
