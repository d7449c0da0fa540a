"""The folded and affine exports at the edges of their launch shapes: warps of
32 points, blocks of 128, one to 18 points per inversion and one to three
blocks per SM (the lengths are those of 152 SMs), with a zero Z in some of
the products.  Exact: every byte against the oracle."""
import ctypes

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


# where the encodings go: pinned memory on a 16-byte boundary is written by the
# kernel itself, past a guard that it leaves alone; any other through a copy
@pytest.mark.parametrize("pinned,shift", [(True, 0), (True, 16), (True, 8), (True, 1), (False, 0)])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 4097, WAVE + 1])
def test_export_destinations(ft, pool, n, pinned, shift):
    torch = pytest.importorskip("torch")
    pts, enc, _ = pool
    idx = np.arange(n) % len(pts)
    a = ft.Array.from_packed(pts).get_subset(idx)
    buf = torch.full((32 * n + 64,), 0xA5, dtype=torch.uint8)
    buf = buf.pin_memory() if pinned else buf
    ft.check(ft.api.lib().ft_array_to_bytes_folded(ctypes.c_void_p(buf.data_ptr() + shift), 32 * n, a.handle))
    out = buf.numpy()
    assert (out[shift:shift + 32 * n].reshape(n, 32) == enc[idx]).all()
    assert (out[:shift] == 0xA5).all() and (out[shift + 32 * n:] == 0xA5).all()


# and where they come from: pinned memory on a 16-byte boundary is read by the
# kernel itself, the rest through a copy; a warp's, a block's and a launch's
# edges, and more points than a launch has threads
@pytest.mark.parametrize("pinned,shift", [(True, 0), (True, 16), (True, 8), (False, 0)])
@pytest.mark.parametrize("n", [1, 33, 129, 8 * WAVE + 1])
def test_decode_sources(ft, pool, n, pinned, shift):
    torch = pytest.importorskip("torch")
    _, enc, _ = pool
    idx = np.arange(n) % len(enc)
    buf = torch.full((32 * n + 64,), 0xA5, dtype=torch.uint8)
    buf = buf.pin_memory() if pinned else buf
    buf.numpy()[shift:shift + 32 * n] = enc[idx].ravel()
    arr, bad = ctypes.c_void_p(), ctypes.c_int64()
    lib = ft.api.lib()
    err = lib.ft_array_from_bytes_folded(ctypes.byref(bad), ctypes.byref(arr), ctypes.c_void_p(buf.data_ptr() + shift), 32 * n)
    want, at = ft.Array.from_bytes_folded(enc[idx])
    assert err == 0 and bad.value == at
    out = np.zeros((n, 32), np.uint8)
    ft.check(lib.ft_array_to_bytes_folded(out.ctypes.data_as(ctypes.c_void_p), out.size, arr))
    lib.ft_array_free(arr)
    assert (out == want.to_bytes_folded()).all()
