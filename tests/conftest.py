import gc
import os
import sys

import numpy as np
import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run with -m gpu on a B200)")


def pytest_collection_modifyitems(config, items):
    if torch.cuda.is_available():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


_pools = []   # (kept: what a test leaves in the framework's caches lives on)


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_call(item):
    """A test that reads how much memory is allocated has an allocator pool of its own: a cached block is handed out whole
    where no more than 1 MB would be left over, so that the figure depends on what earlier tests have left."""
    code = getattr(getattr(item, "function", None), "__code__", None)
    if code is None or "memory_allocated" not in code.co_names or not torch.cuda.is_available():
        yield
        return
    gc.collect()
    _pools.append(torch.cuda.MemPool())
    with torch.cuda.use_mem_pool(_pools[-1]):
        yield


@pytest.fixture(scope="session")
def golden():
    def load(name):
        return np.load(os.path.join(GOLDEN, name))
    return load


def rel_l2(y, ref):
    """||y - ref|| / ||ref|| with fp64 accumulation."""
    y = np.asarray(y, dtype=np.float64)
    ref = np.asarray(ref, dtype=np.float64)
    return float(np.sqrt(((y - ref) ** 2).sum()) / max(np.sqrt((ref ** 2).sum()), 1e-300))
