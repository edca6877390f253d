import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


import pytest


def pytest_configure(config):
    config.addinivalue_line(
        "markers", "gpu: needs a CUDA device (runs the sm_100a kernels)")


@pytest.fixture(params=["rule", "asked"])
def thread_rule(request, monkeypatch):
    """A test with it runs twice: with the threads per dest that lanes_for
    gives the small engines of the tests (eight), and with those that the
    engine was asked for (one by default, as every engine above 50,000
    particles runs)."""
    if request.param == "asked":
        from pysph_b200 import engine
        monkeypatch.setattr(engine, "FILL_THREADS", 0)
