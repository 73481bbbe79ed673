"""pytest configuration: registers the ``gpu`` marker and puts the repository root on ``sys.path``.

Tests marked ``gpu`` call the CUDA library through its C ABI and need a B200; everything else runs on CPU.
"""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run with -m gpu on a B200)")


def plugin_cannot_be_built():
    """True where there is neither a built PJRT plugin nor the OpenXLA header it is compiled against."""
    from __graft_entry__ import _pjrt_include

    plugin = os.path.join(ROOT, "metalhlo_b200", "lib", "pjrt_plugin_metalhlo_b200.so")
    return not os.path.exists(plugin) and _pjrt_include() is None


def pytest_collection_modifyitems(config, items):
    if plugin_cannot_be_built():
        no_plugin = pytest.mark.skip(reason="pjrt_c_api.h is not available here, so the PJRT plugin is not built")
        for item in items:
            if "pjrt" in item.nodeid or item.name.startswith("test_plugin_"):
                item.add_marker(no_plugin)
    try:
        import torch

        has_gpu = torch.cuda.is_available()
    except Exception:  # pragma: no cover
        has_gpu = False
    if has_gpu:
        return
    skip = pytest.mark.skip(reason="no CUDA device in this process")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)
