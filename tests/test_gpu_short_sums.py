"""Sums at the lengths where the one block of quads takes another point each,
and where a launch of many blocks goes before it.  Exact: the oracle's encoding."""
import numpy as np
import pytest

from libftcrypto_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def points(orc):
    g = synth.rng(83)
    return orc.mul(orc.from_scalars(synth.scalars_mod_L(g, 321)), synth.scalars_mod_L(g, 321), threads=8)  # any Z


@pytest.mark.parametrize("n", [0, 2, 3, 4, 8, 9, 32, 33, 63, 64, 65, 128, 129, 256, 257, 319, 320, 321])
def test_sum(ft, orc, points, n):
    a, out = ft.Array.from_packed(points[:n]), ft.Array.init_scalar(2)
    a.reduce_into(out, 1)
    want = orc.encode(orc.reduce(np.ascontiguousarray(points[:n])))
    assert (out.to_bytes_folded() == np.concatenate([orc.encode(orc.zeros(1)), want])).all()
    a.reduce()
    assert len(a) == 1 and (a.to_bytes_folded() == want).all()
