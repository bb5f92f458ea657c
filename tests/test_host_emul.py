"""Host helpers of the library on a stand-in CUDA runtime (tests/host_emul): what they
leave behind when a call fails, which no test may bring about on a GPU."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def emul():
    subprocess.run(["make", "-s", "-C", os.path.join(HERE, "host_emul")], check=True)
    lib = ctypes.CDLL(os.path.join(HERE, "host_emul", "_build", "libhost_emul.so"))
    lib.unitig_buffers.argtypes = [ctypes.c_uint64, ctypes.c_uint64, ctypes.c_uint32]
    lib.side_streams_pass.argtypes = [ctypes.c_uint32, ctypes.c_long, ctypes.POINTER(ctypes.c_long)]
    return lib


@pytest.mark.parametrize("launches", [0, 1, 2, 4, 5, 9])
def test_side_streams_leave_nothing_running(emul, launches):
    """Whichever call of a pass fails, every stream with a launch has been waited for when the pass returns; a pass
    without an error has its launches between the fork and the join."""
    calls = ctypes.c_long()
    assert emul.side_streams_pass(launches, -1, ctypes.byref(calls)) == 0
    for at in range(calls.value):
        assert emul.side_streams_pass(launches, at, ctypes.byref(ctypes.c_long())) == 0, f"call {at} of {calls.value}"


@pytest.mark.parametrize("k", [31, 63, 65, 127])
@pytest.mark.parametrize("n", [0, 1, 1000, 1 << 20])
def test_collation_buffers_know_what_they_hold(emul, n, k):
    """The lm-tigs that the buffers hold are known for the k they are used with, no second call grows them, and a call
    that finds no room leaves none."""
    assert emul.unitig_buffers(n, 2 * n + 5000, k) == 0
