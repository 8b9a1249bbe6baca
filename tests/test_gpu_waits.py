"""Bounded waits of the recursion kernel: rows that never come end the launch with a status, and the context goes on.
tests/native/wave_waits.cpp launches the kernel over a small scenario and leaves one of its tiles out."""

import ctypes
import pathlib
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parents[1]
ALL, STAGED, DIRECT, SHARED, SHORT_RING = range(5)


@pytest.fixture(scope="module")
def waits(tmp_path_factory):
    from cardiotrust_b200 import _lib

    _lib.lib()
    so = tmp_path_factory.mktemp("waits") / "libwave_waits.so"
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I/usr/local/cuda/include",
                           str(ROOT / "tests/native/wave_waits.cpp"), "-o", str(so), str(_lib.LIB_PATH),
                           f"-Wl,-rpath,{_lib.PKG}", "-L/usr/local/cuda/lib64", "-lcudart_static", "-ldl", "-lrt", "-lpthread"])
    lib = ctypes.CDLL(str(so))

    def run(form):
        status, ms = ctypes.c_int(99), ctypes.c_float()
        assert lib.wave_waits(form, ctypes.byref(status), ctypes.byref(ms)) == 0
        return status.value, ms.value

    return run


@pytest.mark.parametrize("form", [STAGED, DIRECT, SHARED], ids=["staged", "direct", "shared"])
def test_rows_that_never_come(waits, form):
    from cardiotrust_b200 import _lib

    status, ms = waits(form)
    assert status == _lib.CT_ERR_TIMEOUT
    assert 1900 < ms < 10000
    assert waits(ALL)[0] == _lib.CT_OK


def test_a_ring_that_could_lose_rows_is_refused(waits):
    """16 rows with delays of 2 to 9, where readers may go back 18 steps: a status at once, nothing runs."""
    from cardiotrust_b200 import _lib

    status, ms = waits(SHORT_RING)
    assert status == _lib.CT_ERR_NOT_SUPPORTED
    assert ms < 100
    assert waits(ALL)[0] == _lib.CT_OK
