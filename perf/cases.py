"""Performance cases: what a program built on this library has it do.

Every case goes through the public entry points, from what the program holds
(host buffers in pinned memory, arrays on the device, a key) to the canonical
32-byte encodings, sums or plaintexts it sends on or stores.

kind        one pass
encrypt     n counters encrypted under a key (ftx_encrypt), both halves exported
scale       n ciphertexts times a secret scalar each (ft_mul of both halves), exported
tally       `vectors` ciphertext vectors of n added to a running total (ftx_ct_add), exported
relay       n received ciphertexts decoded (ft_array_from_bytes_folded), added to a
            total (ftx_ct_add), the total exported
group_sum   n ciphertexts summed by group ("csr": offsets on the device,
            ftx_ct_segmented_sum_csr_device; "isum": keys on the host,
            ft_reduce_isum of both halves), exported
prefix      inclusive or exclusive prefix sums of n ciphertexts (ftx_ct_scan), exported
total       the sum of n ciphertexts (ftx_reduce_into of both halves), exported
decrypt     n ciphertexts of values below m_max (ftx_decrypt)

All arithmetic is exact: the outputs are bytes (canonical encodings) or whole
numbers (plaintexts).
"""
import ctypes
import math

import numpy as np
import torch

import libftcrypto_gb300 as ft
from libftcrypto_gb300 import synth

# 64 32x32-bit products a field multiplication, two operations a product
FIELD_MUL = 128
ADD = 9 * FIELD_MUL         # projective point addition
MIXED_ADD = 7 * FIELD_MUL   # addition of an affine table entry
LADDER = 2340 * FIELD_MUL   # variable-base product by a 253-bit scalar
COMB = 52 * MIXED_ADD       # fixed-base product, radix-32 comb
DECODE = 270 * FIELD_MUL    # a square root
ENCODE = 12 * FIELD_MUL     # 2 products and a share of a batched inversion


def listed():
    return [
        # a client encrypts one form or ballot: latency of a small call
        {"name": "encrypt_16", "kind": "encrypt", "n": 16, "bits": 8},
        # a reporting entity encrypts an account list of a few thousand
        {"name": "encrypt_3001", "kind": "encrypt", "n": 3001, "bits": 16},
        # the bulk encryption of the batched configuration (2^20 8-bit values)
        {"name": "encrypt_1m", "kind": "encrypt", "n": 1 << 20, "bits": 8},
        # a handful of results blinded before they leave: latency
        {"name": "scale_24", "kind": "scale", "n": 24},
        # a mid-size query answer blinded, not a multiple of any tile
        {"name": "scale_5003", "kind": "scale", "n": 5003},
        # the bulk secret-scalar multiplication
        {"name": "scale_512k", "kind": "scale", "n": 1 << 19},
        # 16 parties' vectors of the plain-add configuration's length summed
        {"name": "tally_65536x16", "kind": "tally", "n": 65536, "vectors": 16},
        # an aggregator takes in one party's encoded vector and hands on the total
        {"name": "relay_200003", "kind": "relay", "n": 200003},
        # per-account totals of a transaction table (mean 16 rows a group)
        {"name": "group_sum_4m", "kind": "group_sum", "n": 1 << 22, "groups": 1 << 18, "form": "csr"},
        # running balances over a ledger
        {"name": "prefix_1m", "kind": "prefix", "n": 1000000, "exclusive": False},
        # one grand total over a large table
        {"name": "total_8m", "kind": "total", "n": 1 << 23},
        # the key holder reads the counters of a published table
        {"name": "decrypt_50k", "kind": "decrypt", "n": 50000, "m_max": 65536},
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["encrypt", "scale", "tally", "relay", "group_sum", "prefix", "total", "decrypt"])
    if kind == "encrypt":
        return {"kind": kind, "n": _log(rng, 1, 1 << 20), "bits": rng.choice([1, 8, 16, 32])}
    if kind == "scale":
        return {"kind": kind, "n": _log(rng, 1, 500000)}
    if kind == "tally":
        return {"kind": kind, "n": _log(rng, 100, 200000), "vectors": rng.randint(2, 24)}
    if kind == "relay":
        return {"kind": kind, "n": _log(rng, 50, 400000)}
    if kind == "group_sum":
        n = _log(rng, 2000, 1 << 22)
        return {"kind": kind, "n": n, "groups": max(1, n // rng.randint(3, 50)), "form": rng.choice(["csr", "isum"])}
    if kind == "prefix":
        return {"kind": kind, "n": _log(rng, 500, 1 << 20), "exclusive": rng.random() < 0.3}
    if kind == "total":
        return {"kind": kind, "n": _log(rng, 500, 1 << 23)}
    return {"kind": kind, "n": _log(rng, 1, 100000), "m_max": 1 << rng.randint(8, 16)}


def work(case):
    n, kind = case["n"], case["kind"]
    if kind == "encrypt":
        return {"bytes": n * (8 + 32 + 64), "flops": n * (2 * COMB + 2 * MIXED_ADD + 2 * ENCODE)}
    if kind == "scale":
        return {"bytes": n * (32 + 256 + 256 + 64), "flops": n * (2 * LADDER + 2 * ENCODE)}
    if kind == "tally":
        v = case["vectors"]
        return {"bytes": n * (256 * (v + 2) + 64), "flops": n * (2 * v * ADD + 2 * ENCODE)}
    if kind == "relay":
        return {"bytes": n * (64 + 256 + 256 + 64), "flops": n * (2 * DECODE + 2 * ADD + 2 * ENCODE)}
    if kind == "group_sum":
        g = case["groups"]
        return {"bytes": n * (256 + (8 if case["form"] == "isum" else 0)) + g * (4 + 64), "flops": 2 * n * ADD + 2 * g * ENCODE}
    if kind == "prefix":
        return {"bytes": n * (256 + 256 + 64), "flops": n * (2 * ADD + 2 * ENCODE)}
    if kind == "total":
        return {"bytes": n * 256 + 64, "flops": 2 * n * ADD}
    return {"bytes": n * (256 + 8), "flops": n * (LADDER + ADD + ENCODE)}


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _scalars(g, n):
    """(n, 32) bytes on the GPU: scalars uniform below 2^252 (below the group order)."""
    s = torch.randint(0, 256, (n, 32), dtype=torch.uint8, device="cuda", generator=g)
    s[:, 31] &= 0x0F
    return s


def _values(g, n, hi):
    return torch.randint(0, hi, (n,), dtype=torch.int64, device="cuda", generator=g)


def _pinned(t):
    """A copy in pinned host memory, as a numpy array."""
    return t.cpu().pin_memory().numpy()


def _out(n):
    """Room in pinned host memory for the encodings of n points."""
    return torch.empty((n, ft.FOLDED), dtype=torch.uint8).pin_memory()


def _export(out, array):
    ft.check(ft.api.lib().ft_array_to_bytes_folded(ctypes.c_void_p(out.data_ptr()), out.numel(), array.handle))
    return out


def _key(seed):
    sk = synth.scalars_mod_L(synth.rng(seed), 1)[0]
    return sk, ft.Array.from_scalars(sk[None]).to_bytes_folded()[0]


def _ciphertexts(g, pk, n, hi=256):
    """n ciphertexts of values below hi, on the device, and the values."""
    m, r = _values(g, n, hi), _scalars(g, n)
    c1, c2 = ft.Array.init_scalar(n), ft.Array.init_scalar(n)
    torch.cuda.synchronize()
    ft.encrypt_device(c1, c2, pk, m.data_ptr(), r.data_ptr(), n)
    ft.synchronize()
    return c1, c2, m


def prepare(case, seed):
    ft.init()
    g = _gen(seed)
    sk, pk = _key(seed)
    n, kind = case["n"], case["kind"]
    s = {"kind": kind, "n": n}
    if kind == "encrypt":
        s["pk"], s["bits"] = pk, case["bits"]
        s["m"] = _pinned(_values(g, n, 1 << case["bits"])).view(np.uint64)
        s["r"] = _pinned(_scalars(g, n))
        s["out"] = (_out(n), _out(n))
        return s
    if kind == "decrypt":
        s["c1"], s["c2"], _ = _ciphertexts(g, pk, n, case["m_max"])
        s["sk"], s["m_max"] = sk, case["m_max"]
        return s
    s["c1"], s["c2"], _ = _ciphertexts(g, pk, n)
    rows = n
    if kind == "scale":
        s["k"] = _pinned(_scalars(g, n))
    elif kind == "tally":
        s["parts"] = [_ciphertexts(g, pk, n)[:2] for _ in range(case["vectors"])]
    elif kind == "relay":
        d1, d2, _ = _ciphertexts(g, pk, n)
        s["in"] = tuple(_pinned(torch.from_numpy(d.to_bytes_folded())) for d in (d1, d2))
    elif kind == "group_sum":
        rows, s["form"] = case["groups"], case["form"]
        s["sum"] = (ft.Array.init_scalar(rows), ft.Array.init_scalar(rows))
        if s["form"] == "csr":
            s["offsets"] = torch.from_numpy(synth.csr_offsets(synth.rng(seed), n, rows)).cuda()
        else:
            s["keys"] = _pinned(_values(g, n, rows)).view(np.uint64)
    elif kind == "prefix":
        s["exclusive"] = case["exclusive"]
    elif kind == "total":
        rows = 1
        s["sum"] = (ft.Array.init_scalar(1), ft.Array.init_scalar(1))
    s["out"] = (_out(rows), _out(rows))
    return s


def run(s):
    kind = s["kind"]
    if kind == "decrypt":
        return ft.decrypt(s["c1"], s["c2"], s["sk"], s["m_max"]).view(np.int64)
    if kind == "encrypt":
        a, b = ft.encrypt(s["pk"], s["m"], s["r"], s["bits"])
        return _export(s["out"][0], a), _export(s["out"][1], b)
    a, b = s["c1"], s["c2"]
    if kind == "scale":
        a.mul(s["k"])
        b.mul(s["k"])
    elif kind == "tally":
        for d1, d2 in s["parts"]:
            ft.ct_add(a, b, d1, d2)
    elif kind == "relay":
        (d1, bad1), (d2, bad2) = (ft.Array.from_bytes_folded(x) for x in s["in"])
        ft.ct_add(a, b, d1, d2)
        return _export(s["out"][0], a), _export(s["out"][1], b), bad1, bad2
    elif kind == "group_sum":
        t1, t2 = s["sum"]
        if s["form"] == "csr":
            ft.ct_segmented_sum_csr_device(t1, t2, s["offsets"].data_ptr(), len(t1), a, b)
        else:
            t1.reduce_isum(s["keys"], a)
            t2.reduce_isum(s["keys"], b)
        a, b = t1, t2
    elif kind == "prefix":
        ft.ct_scan(a, b, s["exclusive"])
    else:
        t1, t2 = s["sum"]
        a.reduce_into(t1)
        b.reduce_into(t2)
        a, b = t1, t2
    return _export(s["out"][0], a), _export(s["out"][1], b)


def exact(case, seed):
    """The plaintexts for a decryption; encodings have no value in 64-bit
    arithmetic (they are bytes, the same or wrong)."""
    if case["kind"] != "decrypt":
        return None
    return _values(_gen(seed), case["n"], case["m_max"]).cpu().numpy()
