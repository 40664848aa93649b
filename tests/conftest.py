import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")


def pytest_collection_modifyitems(items):
    """Tests of application binaries that are not there (they are built from sources a
    machine may not have) come last: they fail, and a run that stops at its first
    failure has then run everything else."""
    apps = os.path.join(ROOT, "olive_b200", "_apps")
    if os.path.exists(os.path.join(apps, "BFS")):
        return
    needs = ("_app", "apps_", "dropin", "header_layer")
    items.sort(key=lambda it: any(n in it.nodeid for n in needs))


@pytest.fixture(scope="session")
def golden_dir():
    return GOLDEN
