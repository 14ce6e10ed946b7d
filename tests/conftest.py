import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200); run with -m gpu")
    if not hasattr(config, "workerinput"):  # once, before any worker process loads it
        from tests.emu.emu import build as build_emu
        try:
            build_emu()
        except (OSError, subprocess.CalledProcessError):
            pass  # the tests that need the emulator say why


@pytest.fixture(scope="session", autouse=True)
def _checkers_built():
    """The CPU oracle is built from source if it is missing (no reference sources needed)."""
    if not os.path.exists(os.path.join(ROOT, "oracle", "liboracle.so")):
        subprocess.run(["make", "-s", "-C", os.path.join(ROOT, "oracle"), "oracle"], check=True)
    yield
