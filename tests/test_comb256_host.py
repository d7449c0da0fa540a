"""The radix-256 comb (csrc/comb256.cuh), compiled for the host: digits, table
words split into f16 integers and put together again, signed entries, the first
row's point and the additions, against the oracle's products, and the bound
that the additions' coordinates keep."""
import ctypes
import os
import random
import subprocess

import numpy as np
import pytest

from libftcrypto_gb300 import synth

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def hc(tmp_path_factory, orc):
    so = str(tmp_path_factory.mktemp("comb") / "comb256_host.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared",
                           '-DFT_HOST_EMULATION="../../tests/host/ptx_emul.h"', "-o", so,
                           os.path.join(HERE, "host", "comb256_host.cpp")])
    lib = ctypes.CDLL(so)
    base = orc.from_scalars(synth.int_to_scalar(1)[None])
    lib.hc_comb256_table(base.ctypes.data_as(ctypes.c_void_p))
    return lib


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def test_products(hc, orc):
    vals = [0, 1, 127, 128, 129, 255, 256, 2**255 - 1, 2**255, 2**255 + 12345, 9 * 2**252 - 1, 9 * 2**252, 2**256 - 1,
            synth.L - 1, 8 * synth.L - 1, 8 * synth.L, 8 * synth.L + 1, 0x847777 << 232, 0x877777 << 232, 0x87777777777777777777777777777777 << 128]
    vals += [sum(b << (8 * k) for k in range(31)) for b in (0x7f, 0x80, 0x81)]
    sc = np.concatenate([np.stack([synth.int_to_scalar(v) for v in vals]), synth.scalars_mod_L(synth.rng(7), 100)])
    n = len(sc)
    pts, dig = np.zeros((n, 128), np.uint8), np.zeros((n, 32), np.int32)
    hc.hc_comb256(ptr(pts), ptr(dig), ptr(sc), ctypes.c_size_t(n))
    assert dig[:, :31].min() >= -128 and dig[:, :31].max() <= 127 and dig[:, 31].min() >= 0 and dig[:, 31].max() <= 128
    assert (dig[:, 31] == 128).any()
    assert (orc.encode(pts) == orc.encode(orc.from_scalars(sc))).all()
    assert hc.hc_comb256_tight() == 1


def test_tight_field(hc):
    P = 2**255 - 19
    rnd = random.Random(3)
    edge = [0, 1, 19, P - 1, P, P + 1, 2**255 - 1, 2**255, 2**255 + 1462, 2**256 - 1, 2**256 - 38, 2**256 - 39]
    # operands whose product is just below and above 2^255 (mod p)
    vals = edge + [rnd.getrandbits(256) for _ in range(2000)]
    pairs = [(a, b) for a in edge for b in edge] + [(vals[i], vals[(7 * i + 5) % len(vals)]) for i in range(len(vals))]
    pairs += [(x, pow(x, -1, P) * t % P) for x in vals[12:200] for t in (P - 1, P - 2, P - 1462, 1, 2, 1443, 1444)]
    buf = [ctypes.create_string_buffer(32) for _ in range(3)]
    for a, b in pairs:
        assert hc.hc_comb256_field(a.to_bytes(32, "little"), b.to_bytes(32, "little"), *buf) == 1
        prod, total, diff = (int.from_bytes(x.raw, "little") for x in buf)
        assert prod % P == a * b % P and total % P == 2 * a * b % P and diff % P == (a - b) % P


@pytest.mark.parametrize("bits", [1, 7, 8, 15, 16, 31, 32, 63, 64])
def test_small_values(hc, orc, bits):
    top = (1 << bits) - 1
    g = synth.rng(bits)
    m = np.array([0, 1, top, top // 2, top - top // 3] + [int(x) & top for x in g.integers(0, 2**63, 20)], np.uint64)
    pts = np.zeros((len(m), 128), np.uint8)
    hc.hc_comb256_small(ptr(pts), ptr(m), ctypes.c_size_t(len(m)), bits)
    assert (orc.encode(pts) == orc.encode(orc.from_scalars(orc.small_to_scalars(m)))).all()
