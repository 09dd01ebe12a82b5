import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA (B200) device")


def _skip_without_reference(e):
    """Tests against the compiled reference need what is built from its sources
    (oracle/_ref, the C++ overloads and their drivers). Where neither those
    sources nor the built libraries are there, such a test is skipped; with the
    sources there, a library that is missing or does not load is a failure."""
    import __graft_entry__
    if os.path.isdir(os.path.join(__graft_entry__.REFERENCE, "src")):
        return
    text = str(e)
    if isinstance(e, OSError) and "oracle/_ref/" in text and "No such file" in text or \
            isinstance(e, AssertionError) and "not built (make" in text:
        pytest.skip("needs libraries built from the reference's sources, which are not here")


@pytest.hookimpl(wrapper=True)
def pytest_runtest_setup(item):
    try:
        return (yield)
    except (OSError, AssertionError) as e:
        _skip_without_reference(e)
        raise


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    try:
        return (yield)
    except (OSError, AssertionError) as e:
        _skip_without_reference(e)
        raise


@pytest.fixture(scope="session")
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")
