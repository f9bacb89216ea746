import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); parity tests through the C ABI")


def have_gpu() -> bool:
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


def pytest_collection_modifyitems(config, items):
    if have_gpu():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for it in items:
        if "gpu" in it.keywords:
            it.add_marker(skip)


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_call(item):
    """A test of the compiled reference, where that is not built (it is made
    from the reference's sources, which need not be at hand), is skipped."""
    outcome = yield
    err = outcome.excinfo[1] if outcome.excinfo else None
    ref = os.path.join("oracle", "_ref")
    if isinstance(err, FileNotFoundError) and ref in str(err) and not os.path.isdir(os.path.join(ROOT, ref)):
        outcome.force_exception(pytest.skip.Exception(f"no compiled reference: {err}"))
