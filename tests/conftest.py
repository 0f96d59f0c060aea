"""pytest config: `gpu` marker + import paths (repo root for `oracle`, the package dir for
the drop-in modules and `pg_b200`)."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "multimodal-financial-analysis-tool-using-paligemma_b200")
for p in (PKG, ROOT):
    if p not in sys.path:
        sys.path.insert(0, p)
GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box)")
    config.addinivalue_line("markers", "slow: full-size model, minutes of CPU oracle time")


def pytest_collection_modifyitems(config, items):
    import torch
    if torch.cuda.is_available():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for it in items:
        if "gpu" in it.keywords:
            it.add_marker(skip)


@pytest.fixture(scope="session")
def golden_dir():
    return GOLDEN


@pytest.fixture
def gemm_workspace():
    """80 MB of scratch for the split products (pg_set_workspace) for one test; then the process's own again: the engines', or none."""
    import torch
    from pg_b200 import _cabi as cabi
    from pg_b200.engine import _WORKSPACES
    L, ws = cabi.lib(), torch.empty(80 << 20, dtype=torch.uint8, device="cuda")
    cabi.check(L.pg_set_workspace(ws.data_ptr(), ws.numel()))
    yield ws
    torch.cuda.synchronize()
    own = [w for w in _WORKSPACES.values() if w.device.index == torch.cuda.current_device()]   # the engines' key may name no index
    cabi.check(L.pg_set_workspace(own[-1].data_ptr(), own[-1].numel()) if own else L.pg_set_workspace(None, 0))
