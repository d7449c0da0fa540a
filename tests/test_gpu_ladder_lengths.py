"""ft_mul and ft_scale at the lengths where the ladder's launch changes (with
152 SMs): four lanes per point up to 160 points per SM, the 224-thread kernel, four
lanes again up to 256, whole waves of 384 with a rest in a second launch.  Exact:
the oracle's coordinates, word for word, edge scalars among them."""
import numpy as np
import pytest

from libftcrypto_gb300 import synth

pytestmark = pytest.mark.gpu

SM = 152


@pytest.fixture(scope="module")
def pool(orc):
    """251 points (one off the curve), 251 scalars, all products by pairs (i, i)."""
    g = synth.rng(71)
    n = 251
    pts = orc.mul(orc.from_scalars(synth.scalars_mod_L(g, n), threads=8), synth.scalars_mod_L(g, n), threads=8)
    pts[7] = g.integers(0, 256, 128, dtype=np.uint8)
    k = synth.scalars_mod_L(g, n)
    for i, x in enumerate([0, 1, 8, 15, 16, synth.L - 1, 2**255 - 1, 2**255 + 12345, 2**256 - 1]):
        k[20 + i] = synth.int_to_scalar(x)
    return pts, k, orc.mul(pts, k, threads=8), orc.mul(pts, np.repeat(k[:1], n, axis=0), threads=8)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 33, 32 * SM + 1, 96 * SM + 1, 160 * SM, 160 * SM + 1, 224 * SM + 1, 256 * SM + 1,
                               384 * SM, 384 * SM + 1, (384 + 160) * SM + 5, (384 + 256) * SM + 1])
def test_lengths(ft, pool, n):
    pts, k, products, scaled = pool
    idx = np.arange(n) % len(pts)
    base = ft.Array.from_packed(pts)
    a = base.get_subset(idx)
    a.mul(k[idx])
    assert (a.to_packed() == products[idx]).all()
    b = base.get_subset(idx)
    b.scale(k[0])
    assert (b.to_packed() == scaled[idx]).all()
