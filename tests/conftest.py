"""Shared test setup: import paths, the `gpu` marker, and device guards."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for sub in ("sgemm.cu_b200", "oracle"):
    p = os.path.join(ROOT, sub)
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a B200 (sm_100a) GPU")


def _have_gpu() -> bool:
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


def pytest_collection_modifyitems(config, items):
    if _have_gpu():
        # Without the build of the reference's own kernels the GPU tests against them
        # fail: after all others, so that a run that stops at its first failure has
        # run everything else.
        if not os.path.exists(os.path.join(ROOT, "oracle", "_ref", "libref_sgemm.so")):
            items.sort(key=lambda i: "gpu" in i.keywords and "reference" in i.nodeid)
        return
    skip = pytest.mark.skip(reason="no CUDA device in this environment")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)
