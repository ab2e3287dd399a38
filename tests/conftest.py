import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (runs on the B200)")


def pytest_collection_modifyitems(items):
    """Tests that step the reference itself are skipped where its library was
    not built (its sources are not there), those too that do not say so."""
    from oracle.oracle import ref_available
    if not ref_available():
        for item in items:
            code = getattr(getattr(item, "function", None), "__code__", None)
            if code is not None and "RefSim" in code.co_names:
                item.add_marker(pytest.mark.skip(reason="oracle/_ref not built"))
