import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (sm_103a) and the built CUDA library")
    config.addinivalue_line("markers", "slow: longer-running parity cases")


def gpu_available() -> bool:
    try:
        import torch

        return torch.cuda.is_available()
    except Exception:
        return False


@pytest.fixture(scope="session")
def goldens():
    import json

    with open(os.path.join(ROOT, "tests", "golden", "reference_goldens.json")) as f:
        return json.load(f)


@pytest.fixture(autouse=True)
def _library_defaults(request):
    """Tests that set the process-wide scheduling leave the library's defaults behind."""
    yield
    if request.node.get_closest_marker("gpu"):
        from galax_gb300 import _lib

        L = _lib.load()
        _lib.check(L.gal_set_team(-1), "gal_set_team")
        _lib.check(L.gal_set_split_fraction(0.1), "gal_set_split_fraction")
        _lib.check(L.gal_set_table_lanes(0), "gal_set_table_lanes")
