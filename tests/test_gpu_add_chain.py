"""Additions queued one after another on the same arrays, each reading what the
one before wrote, with nothing in between that waits: the launches overlap at
their ends, at lengths of one block, a few, and more than are resident at once.
Exact: every output's encoding against
the oracle's."""
import os

import numpy as np
import pytest

from libftcrypto_gb300 import synth

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 1


@pytest.mark.parametrize("n", [1, 128, 129, 70001])
def test_add_chain(ft, orc, n):
    g = synth.rng(91)
    base = orc.from_scalars(synth.scalars_mod_L(g, 997), threads=THREADS)
    a, b, c, d = (np.ascontiguousarray(base[(np.arange(n) * 5 + k) % len(base)]) for k in range(4))
    A, B, C, D = (ft.Array.from_packed(x) for x in (a, b, c, d))
    for _ in range(4):
        ft.ct_add(A, B, C, D)
        ft.ct_sub(C, D, B, A)
        A.add(D)
        B.sub(A)
    for _ in range(4):
        a, b = orc.add(a, c, THREADS), orc.add(b, d, THREADS)
        c, d = orc.sub(c, b, THREADS), orc.sub(d, a, THREADS)
        a = orc.add(a, d, THREADS)
        b = orc.sub(b, a, THREADS)
    for got, want in ((A, a), (B, b), (C, c), (D, d)):
        assert (got.to_bytes_folded() == orc.encode(want, THREADS)).all()
