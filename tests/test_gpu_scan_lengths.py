"""Scans and sums at the lengths where their launches change (with 152 SMs):
one block, block scans of the points themselves, sums of 4 and more points per
thread in one wave and two, more than one point per thread of the block scans;
quads alone and after the first pass.  Exact: every output's encoding against
the oracle's."""
import os

import numpy as np
import pytest

from libftcrypto_gb300 import synth

pytestmark = pytest.mark.gpu

SM, THREADS = 152, os.cpu_count() or 1


@pytest.fixture(scope="module")
def points(orc):
    g = synth.rng(81)
    base = orc.from_scalars(synth.scalars_mod_L(g, 4099), threads=THREADS)
    return orc.mul(base, synth.scalars_mod_L(g, 4099), threads=THREADS)  # any Z


def take(points, n, first):
    return np.ascontiguousarray(points[(np.arange(n) * 7 + first) % len(points)])


@pytest.mark.parametrize("n", [1, 2, 64, 65, 512, 513, 4097, 128 * SM, 128 * SM + 1, 256 * SM, 256 * SM + 1,
                               4 * 384 * SM // 2 + 3, 40 * 384 * SM // 2 + 2])
def test_scan_lengths(ft, orc, points, n):
    a, b = take(points, n, 0), take(points, n, 5)
    for exclusive in (False, True):
        wa = orc.encode(orc.scan(a, exclusive, threads=THREADS), THREADS)
        wb = orc.encode(orc.scan(b, exclusive, threads=THREADS), THREADS)
        A, B, C = ft.Array.from_packed(a), ft.Array.from_packed(b), ft.Array.from_packed(a)
        ft.ct_scan(A, B, exclusive)
        assert (A.to_bytes_folded() == wa).all()
        assert (B.to_bytes_folded() == wb).all()
        C.prescan() if exclusive else C.scan()
        assert (C.to_bytes_folded() == wa).all()


@pytest.mark.parametrize("n", [1, 31, 33, 32 * SM, 32 * SM + 1, 512 * SM, 512 * SM + 1, 1024 * SM + 77])
def test_sum_lengths(ft, orc, points, n):
    a = take(points, n, 1)
    A, out = ft.Array.from_packed(a), ft.Array.init_scalar(3)
    A.reduce_into(out, 1)
    want = orc.encode(orc.reduce(a, threads=THREADS))
    assert (out.to_bytes_folded()[1:2] == want).all()
    A.reduce()
    assert len(A) == 1 and (A.to_bytes_folded() == want).all()
