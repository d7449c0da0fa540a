"""Which host buffers a kernel addresses itself (csrc/host_view.h), over
made-up maps of pinned memory: all of a buffer in one block, aligned, or not at
all."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PAGE = 65536


@pytest.fixture(scope="module")
def view(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("view") / "host_view_host.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", so,
                           os.path.join(HERE, "host", "host_view_host.cpp")])
    f = ctypes.CDLL(so).hv_device_view
    U = ctypes.c_uint64
    f.restype, f.argtypes = U, [ctypes.POINTER(U), ctypes.POINTER(U), ctypes.c_int, U, U, U]

    def run(blocks, p, n, shift=0):
        a = (U * len(blocks))(*[b[0] for b in blocks])
        s = (U * len(blocks))(*[b[1] for b in blocks])
        return f(a, s, len(blocks), shift, p, n)
    return run


def test_within_a_block(view):
    block = [(16 * PAGE, 4 * PAGE)]
    for p, n in [(16 * PAGE, 4 * PAGE), (16 * PAGE, 1), (20 * PAGE - 32, 32), (16 * PAGE + 48, 3 * PAGE)]:
        assert view(block, p, n) == p
    assert view(block, 16 * PAGE, 64, shift=1 << 40) == 16 * PAGE + (1 << 40)
    for p, n in [(16 * PAGE + 8, 32), (16 * PAGE + 1, 32), (15 * PAGE, 32), (20 * PAGE, 32)]:
        assert view(block, p, n) == 0


@pytest.mark.parametrize("p, n", [(16 * PAGE, 4 * PAGE + 1), (20 * PAGE - 32, 64), (15 * PAGE, 2 * PAGE),
                                  (16 * PAGE + 16, 2**64 - 32 * PAGE)])
def test_past_a_block(view, p, n):
    assert view([(16 * PAGE, 4 * PAGE)], p, n) == 0


@pytest.mark.parametrize("gap", [1, 16, PAGE, 3 * PAGE])
def test_pages_between_two_blocks(view, gap):
    blocks = [(16 * PAGE, PAGE), (17 * PAGE + gap, PAGE)]
    for p, n in [(16 * PAGE, 2 * PAGE + gap), (17 * PAGE - 32, gap + 64), (17 * PAGE - 16, gap + 17)]:
        assert view(blocks, p, n) == 0
    assert view(blocks, 16 * PAGE, PAGE) == 16 * PAGE
