import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (ROOT, os.path.join(ROOT, "oracle"), os.path.join(ROOT, "tests")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); runs the CUDA path")
    config.addinivalue_line("markers", "slow: long-running test")


def pytest_collection_modifyitems(config, items):
    try:
        import torch
        has_gpu = torch.cuda.is_available()
    except Exception:
        has_gpu = False
    if has_gpu:
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for it in items:
        if "gpu" in it.keywords:
            it.add_marker(skip)


@pytest.fixture(params=[1, 0], ids=["clusters", "grid"])
def krylov_mode(request):
    """Both launch forms of the Krylov solves on a domain of few small systems: clusters (the default choice, one cluster
    per system on chip) and the persistent grid."""
    from pict_b200 import _lib
    lib = _lib.load()
    lib.pict_krylov_set_cluster_mode(request.param)
    yield request.param
    lib.pict_krylov_set_cluster_mode(1)
