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


@pytest.mark.parametrize("n", [1, 33, 96 * SM, 96 * SM + 1])
def test_short_arrays_at_the_same_time(ft, orc, pool, n):
    """Short arrays are multiplied beside each other: twice in a row, with the
    scalars' pinned buffer refilled after each call, a length change and an
    addition of one to the other in between, exports and a free right after."""
    torch = pytest.importorskip("torch")
    pts, k, _, _ = pool
    i1, i2 = np.arange(n) % len(pts), (np.arange(n) * 5 + 3) % len(pts)
    hk = torch.empty((n, 32), dtype=torch.uint8).pin_memory().numpy()
    a, b = ft.Array.from_packed(pts[i1]), ft.Array.from_packed(pts[i2])
    wa, wb = pts[i1], pts[i2]
    for turn in range(3):
        for arr in (a, b):
            hk[:] = k[(np.arange(n) + 7 * turn + (arr is b)) % len(k)]
            arr.mul(hk)
            hk[:] = 255  # the caller's own again
        wa = orc.mul(wa, k[(np.arange(n) + 7 * turn) % len(k)], threads=8)
        wb = orc.mul(wb, k[(np.arange(n) + 7 * turn + 1) % len(k)], threads=8)
        if turn == 1:
            a.add(b)
            wa = orc.add(wa, wb, threads=8)
    c = ft.Array.from_packed(pts[i1])
    c.add(a)
    assert (a.to_packed() == wa).all()
    assert (b.to_packed() == wb).all()
    hk[:] = k[np.arange(n) % len(k)]
    b.mul(hk)
    b.set_length(n // 2)
    wb = orc.mul(wb, k[np.arange(n) % len(k)], threads=8)
    assert (b.to_packed() == wb[:n // 2]).all()
    a.mul(hk)
    a.free()
    assert (c.to_packed() == orc.add(pts[i1], wa, threads=8)).all()
