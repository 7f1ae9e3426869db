import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200); runs the CUDA library")


@pytest.fixture(scope="session")
def oracle():
    from oracle import oracle as O
    O.build()
    return O


@pytest.fixture(scope="session")
def cad():
    import cutanddisplacejulia_b200 as cad
    from cutanddisplacejulia_b200 import build
    build.build()
    return cad


@pytest.fixture
def fresh_context(cad, monkeypatch):
    """A context of the test's own in the process-wide one's place (no
    workspace grown by earlier tests)."""
    import ctypes

    from cutanddisplacejulia_b200 import _lib
    L, h = _lib.load(), ctypes.c_void_p()
    _lib.check(L.cad_init(0, ctypes.byref(h)), None)
    monkeypatch.setitem(_lib._ctx, 0, h)
    yield h
    L.cad_destroy(h)
