"""A sweep's launch reports its own failure once and leaves nothing for the next launch's check."""
import ctypes
import os
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def launch():
    out = os.path.join(tempfile.mkdtemp(), "launch_host.so")
    subprocess.run(["/usr/bin/g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I/usr/local/cuda/include",
                    "-o", out, os.path.join(HERE, "host", "launch_host.cpp")], check=True)
    return ctypes.CDLL(out).host_launch


@pytest.mark.parametrize("error", [0, 9, 2])        # success, invalid configuration, out of memory
def test_a_failed_launch_leaves_no_error_behind(launch, error):
    left, seen = ctypes.c_int(-1), ctypes.c_int(-1)
    assert launch(error, ctypes.byref(left), ctypes.byref(seen)) == error
    assert seen.value == 71
    assert left.value == 0
