import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.join(ROOT, "oracle"))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200) and the built extension")


def pytest_collection_modifyitems(config, items):
    """A GPU test that takes far longer than any does (the slowest some
    seconds) ends with every thread's stack instead of holding the GPU."""
    if config.pluginmanager.hasplugin("timeout"):
        for item in items:
            if item.get_closest_marker("gpu") and not item.get_closest_marker("timeout"):
                item.add_marker(pytest.mark.timeout(240, method="thread"))


@pytest.fixture(autouse=True)
def bounded_waits(request, monkeypatch):
    """Runners that the scheduling tests make without a wait limit get one of
    a minute: one of them has twice waited until it was killed."""
    if request.module.__name__ == "test_gpu_batch":
        from goav1_b200.postfilter import PostFilterRunner

        monkeypatch.setattr(PostFilterRunner.__init__, "__defaults__", (0, False, 60_000_000))


@pytest.fixture(scope="session")
def oracle():
    import oracle_ctypes

    return oracle_ctypes.lib()


@pytest.fixture(scope="session")
def kats():
    import json

    with open(os.path.join(ROOT, "tests", "golden", "kats.json")) as f:
        return json.load(f)
