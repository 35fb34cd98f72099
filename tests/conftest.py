import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "efwi-3d_b200")
for p in (ROOT, PKG):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200)")


def cuda_ok():
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


@pytest.fixture(autouse=True)
def _reference_checker(monkeypatch):
    """Tests that compare with the reference's own kernels compiled for the CPU
    are skipped where its sources are not there to build them from."""
    import oracle
    if not oracle.ref_available():
        monkeypatch.setattr(oracle, "ref", lambda: pytest.skip(
            "oracle/_ref is not built: the reference's sources are not here"))
