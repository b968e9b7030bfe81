import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
for p in (ROOT / "wavefront-path-tracer_b200", ROOT / "oracle"):
    if str(p) not in sys.path:
        sys.path.insert(0, str(p))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200)")


@pytest.fixture(scope="session")
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("GPU test run without a CUDA device")
    torch.zeros(1, device="cuda")
    return torch


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    """A comparison with the reference's own build skips where that has not
    been built (oracle/Makefile; needs the reference's sources), whether the
    test or a child process of it finds the library missing."""
    try:
        return (yield)
    except (FileNotFoundError, AssertionError) as e:
        if "not built (make -C oracle)" in str(e):
            pytest.skip("the reference's libraries are not built (make -C oracle)")
        raise
