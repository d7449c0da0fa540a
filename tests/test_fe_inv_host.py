"""The division-step inversion (csrc/fe_inv.cuh), compiled for the host,
against Python's modular inverse: canonical results for loosely reduced
inputs, 0 for 0."""
import ctypes
import os
import random
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
P = 2**255 - 19


@pytest.fixture(scope="module")
def inv(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("inv") / "fe_inv_host.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fsanitize=undefined",
                           "-fno-sanitize-recover=undefined",
                           '-DFT_HOST_EMULATION="../../tests/host/ptx_emul.h"', "-o", so,
                           os.path.join(HERE, "host", "fe_inv_host.cpp")])
    lib = ctypes.CDLL(so)

    def run(vals):
        z = np.frombuffer(b"".join(x.to_bytes(32, "little") for x in vals), np.uint32).copy()
        out = np.zeros_like(z)
        lib.hi_fe_inv(out.ctypes.data_as(ctypes.c_void_p), z.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(len(vals)))
        return [int.from_bytes(out[8 * i:8 * i + 8].tobytes(), "little") for i in range(len(vals))]
    return run


def test_inverse(inv):
    rnd = random.Random(1)
    vals = [0, 1, 2, 3, 19, 38, P - 1, P - 2, P, P + 1, (P + 1) // 2, 2 * P - 1, 2 * P, 2 * P + 1, 2**255 - 1, 2**255,
            2**256 - 1]
    vals += [2**k for k in range(256)] + [2**k - 1 for k in range(1, 257)] + [P - 2**k for k in range(255)]
    vals += [pow(2**k, -1, P) for k in range(256)]
    vals += [rnd.getrandbits(256) for _ in range(20000)] + [rnd.getrandbits(rnd.randint(1, 255)) for _ in range(5000)]
    got = inv(vals)
    for v, h in zip(vals, got):
        assert h == (pow(v, P - 2, P) if v % P else 0), hex(v)
