"""Fixed-base products at the lengths where the comb's launch changes (with 152
SMs, in ciphertexts; products of B alone at twice as many): clusters of eight,
four and two blocks to a tile of 128 up to a quarter, a half and a whole of a tile
per SM, then tiles of 256 and 384 by what takes fewer rounds.  Exact: the
oracle's encodings, edge scalars among them."""
import numpy as np
import pytest

from libftcrypto_gb300 import synth

pytestmark = pytest.mark.gpu

SM = 152
EDGES = [SM // 8 * 128, SM // 4 * 128, SM // 2 * 128, SM // 2 * 256, SM // 2 * 384, 2 * (SM // 2) * 256, 2 * (SM // 2) * 384]
LENGTHS = sorted([1, 127, 128, 129] + EDGES + [n + 1 for n in EDGES])


@pytest.fixture(scope="module")
def pool(ft, orc):
    """251 nonces and plaintexts, their encryptions and two fresh nonces' worth
    of re-randomisation as the oracle has them."""
    g = synth.rng(73)
    n = 251
    r, r2 = synth.scalars_mod_L(g, n), synth.scalars_mod_L(g, n)
    for i, x in enumerate([0, 1, 128, synth.L - 1, 8 * synth.L - 1, 8 * synth.L, 2**255 - 1, 2**255 + 12345, 2**256 - 1]):
        r[10 + i] = r2[200 - i] = synth.int_to_scalar(x)
    m = g.integers(0, 256, n, dtype=np.uint64)
    m[:4] = [0, 255, 128, 127]
    big = g.integers(0, 2**64 - 1, n, dtype=np.uint64)
    big[:5] = [0, 1, 128, 2**63, 2**64 - 1]
    pk = orc.from_scalars(synth.scalars_mod_L(g, 1))
    pks = np.repeat(pk, n, axis=0)
    c1, c2 = orc.from_scalars(r), orc.add(orc.from_scalars(orc.small_to_scalars(m)), orc.mul(pks, r, threads=8))
    d1, d2 = orc.add(c1, orc.from_scalars(r2)), orc.add(c2, orc.mul(pks, r2, threads=8))
    enc = {k: orc.encode(v) for k, v in dict(c1=c1, c2=c2, d1=d1, d2=d2, small=orc.from_scalars(orc.small_to_scalars(big))).items()}
    return {"r": r, "r2": r2, "m": m, "big": big, "pk": orc.encode(pk)[0], **enc}


def same(a, want, idx):
    got = a.to_bytes_folded()
    return got.shape[0] == len(idx) and (got == want[idx]).all()


@pytest.mark.parametrize("n", LENGTHS)
def test_ciphertexts(ft, pool, n):
    torch = pytest.importorskip("torch")
    i = np.arange(n) % 251
    d_m = torch.from_numpy(pool["m"].view(np.int64)[i]).cuda()
    d_r, d_r2 = torch.from_numpy(pool["r"][i]).cuda(), torch.from_numpy(pool["r2"][i]).cuda()
    torch.cuda.synchronize()
    c1, c2 = ft.Array.init_scalar(n), ft.Array.init_scalar(n)
    ft.encrypt_device(c1, c2, pool["pk"], d_m.data_ptr(), d_r.data_ptr(), n, 8)
    assert same(c1, pool["c1"], i) and same(c2, pool["c2"], i)
    ft.rerandomise_device(c1, c2, pool["pk"], d_r2.data_ptr(), n)
    assert same(c1, pool["d1"], i) and same(c2, pool["d2"], i)


@pytest.mark.parametrize("n", [2 * k for k in EDGES] + [2 * k + 1 for k in EDGES])
def test_products_of_the_base_point(ft, pool, n):
    i = np.arange(n) % 251
    assert same(ft.Array.from_scalars(pool["r"][i]), pool["c1"], i)
    assert same(ft.Array.from_small_scalars(pool["big"][i]), pool["small"], i)


# one pass of the grid: where ftx_encrypt cuts its inputs in two
@pytest.mark.parametrize("n", [SM * 384 // 2 - 1, SM * 384 // 2, SM * 384 // 2 + 1])
def test_host_inputs_at_the_cut(ft, pool, n):
    i = np.arange(n) % 251
    m, r = pool["m"][i], pool["r"][i]
    c1, c2 = ft.encrypt(pool["pk"], m, r, 8)
    assert same(c1, pool["c1"], i) and same(c2, pool["c2"], i)
    for at in (0, n - 1):
        bad = m.copy()
        bad[at] = 256
        with pytest.raises(ft.FtError) as e:
            ft.encrypt(pool["pk"], bad, r, 8)
        assert e.value.code == 3
