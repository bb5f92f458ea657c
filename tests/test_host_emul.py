"""Host helpers of the library on a stand-in CUDA runtime (tests/host_emul): what they
leave behind when a call fails, which no test may bring about on a GPU."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import test_parse_emul as host_parse
from test_gpu_parse import fasta_text, fastq_text

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def emul():
    subprocess.run(["make", "-s", "-C", os.path.join(HERE, "host_emul"), "_build/libhost_emul.so"], check=True)
    lib = ctypes.CDLL(os.path.join(HERE, "host_emul", "_build", "libhost_emul.so"))
    lib.unitig_buffers.argtypes = [ctypes.c_uint64, ctypes.c_uint64, ctypes.c_uint32]
    lib.parse_state_bytes.restype = ctypes.c_uint64
    lib.parse_state_bytes.argtypes = [ctypes.c_uint64]
    lib.side_streams_pass.argtypes = [ctypes.c_uint32, ctypes.c_long, ctypes.POINTER(ctypes.c_long)]
    return lib


@pytest.fixture(scope="module")
def route():
    subprocess.run(["make", "-s", "-C", os.path.join(HERE, "host_emul"), "_build/libparse_route.so"], check=True)
    lib = ctypes.CDLL(os.path.join(HERE, "host_emul", "_build", "libparse_route.so"))
    lib.parse_emul.restype = ctypes.c_int
    lib.parse_emul.argtypes = [ctypes.c_char_p, ctypes.c_uint64, ctypes.c_int, ctypes.c_uint32,
                               ctypes.POINTER(host_parse.U64P), host_parse.U64P, ctypes.POINTER(host_parse.U64P),
                               ctypes.POINTER(host_parse.U32P), host_parse.U64P]
    lib.parse_emul_free.argtypes = [ctypes.c_void_p]
    return lib


@pytest.mark.parametrize("launches", [0, 1, 2, 4, 5, 9])
def test_side_streams_leave_nothing_running(emul, launches):
    """Whichever call of a pass fails, every stream with a launch has been waited for when the pass returns; a pass
    without an error has its launches between the fork and the join."""
    calls = ctypes.c_long()
    assert emul.side_streams_pass(launches, -1, ctypes.byref(calls)) == 0
    for at in range(calls.value):
        assert emul.side_streams_pass(launches, at, ctypes.byref(ctypes.c_long())) == 0, f"call {at} of {calls.value}"


@pytest.mark.parametrize("launches", [0, 1, 2, 3, 4, 9])
def test_side_streams_are_made_when_used(emul, launches):
    """A context, or a run with one table class, pays for no stream; every one is made once."""
    assert emul.side_streams_made(launches) == min(3, max(0, launches - 1))


@pytest.mark.parametrize("k", [31, 63, 65, 127])
@pytest.mark.parametrize("n", [0, 1, 1000, 1 << 20])
def test_collation_buffers_know_what_they_hold(emul, n, k):
    """The lm-tigs that the buffers hold are known for the k they are used with, no second call grows them, and a call
    that finds no room leaves none."""
    assert emul.unitig_buffers(n, 2 * n + 5000, k) == 0


@pytest.mark.parametrize("size", [1 << 20, 640_000_000, 3_060_000_000])
def test_parse_state_stays_small(emul, size):
    """The parser's state per byte of text: 3/8 of a byte of device memory, plus the buffers' quarter of headroom."""
    assert 0 < emul.parse_state_bytes(size) <= size * 3 // 8 * 5 // 4 + (1 << 17)


@pytest.mark.parametrize("case", range(7))
def test_parse_by_stored_words(route, case):
    """The parser's passes by the words they leave for each other (a group's function, then its emissions; bases and
    breaks before every 32 groups): the host packer's stream and fragments."""
    rng = np.random.default_rng(700 + case)
    if case < 3:
        k = [31, 63, 15][case]
        host_parse.check(route, fasta_text(rng, k, int(rng.integers(1, 12)), 30_000), k)
    elif case < 5:
        host_parse.check(route, fastq_text(rng, 31, int(rng.integers(50, 3_000))), 31)
    else:
        host_parse.test_edge_texts(route) if case == 5 else host_parse.test_fasta_long_lines_and_crlf(route)


def test_machines_are_held_to_what_the_word_steps_assume(route):
    """The compile-time check of the parser's machines tells exactly those whose runs the word-wise steps read rightly."""
    assert route.runs_alike_mismatches() == 0
