import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (ROOT, os.path.join(ROOT, "oracle")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); runs the CUDA path")


def pytest_collection_modifyitems(items):
    """Tests that want the reference's compiled code come last: where its source is absent
    they fail, and a run that stops at the first failure has then run all the others."""
    wants_ref = lambda i: "_need_ref" in i.function.__code__.co_names
    items.sort(key=wants_ref)


@pytest.fixture(scope="session")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("GPU test selected but no CUDA device is visible")
    from ed_solver_b200 import edk
    c = edk.Context(0)
    yield c
    c.close()


@pytest.fixture(autouse=True)
def _default_launch_mode(request):
    """The session's context leaves every test in the launch mode that users get."""
    yield
    if "ctx" in request.fixturenames:
        request.getfixturevalue("ctx").set_graphs(False)
