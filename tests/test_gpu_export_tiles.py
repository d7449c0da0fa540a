"""The folded and affine exports at the edges of their launch shapes: warps of
32 points, blocks of 128, one to 18 points per inversion and one to three
blocks per SM (the lengths are those of 152 SMs), with a zero Z in some of
the products.  Exact: every byte against the oracle."""
import numpy as np
import pytest

from libftcrypto_gb300 import synth

pytestmark = pytest.mark.gpu

WAVE = 152 * 128


@pytest.fixture(scope="module")
def pool(orc):
    g = synth.rng(61)
    pts = orc.mul(orc.from_scalars(synth.scalars_mod_L(g, 509), threads=8), synth.scalars_mod_L(g, 509), threads=8)
    pts[100] = 0  # Z = 0
    return pts, orc.encode(pts), orc.to_affine(pts)


@pytest.mark.parametrize("n", [1, 31, 33, 128, 129, WAVE, WAVE + 1, 2 * WAVE - 31, 18 * WAVE, 18 * WAVE + 1,
                               36 * WAVE + 1, 54 * WAVE + 33])
def test_export_lengths(ft, pool, n):
    pts, enc, aff = pool
    idx = np.arange(n) % len(pts)
    a = ft.Array.from_packed(pts).get_subset(idx)
    assert (a.to_bytes_folded() == enc[idx]).all()
    assert (a.to_bytes_affine() == aff[idx]).all()
