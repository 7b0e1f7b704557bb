import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box)")


@pytest.fixture(scope="session")
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.set_device(0)
    return torch.device("cuda:0")


@pytest.fixture(autouse=True)
def _without_reference_kernels(monkeypatch):
    """The bit oracle is built from the reference's kernel sources; where they were not there to build it from, a test that asks for it is skipped."""
    from oracle import ref_cpu
    if not ref_cpu.available():
        monkeypatch.setattr(ref_cpu, "lib", lambda: pytest.skip("reference kernels not built (oracle/Makefile)"))
