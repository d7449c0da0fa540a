"""The word that a kernel sets when a wait with a limit runs out.  Whatever was
computed since may be invalid, so no call may answer from it: each call reports
it when it begins, and a call that waits for the GPU reports it when it has
waited, for a kernel queued before may have set it meanwhile.  No kernel fails
here: the host sets the word (mapped host memory)."""
import ctypes
import threading

import numpy as np
import pytest

from libftcrypto_gb300 import synth

pytestmark = pytest.mark.gpu

INTERNAL, TIMEOUT = 9, 702


@pytest.fixture
def word(ft):
    address = ft.api.lib()["_ZN2ft10fault_wordEv"]  # ft::fault_word(), internal.h
    address.restype = ctypes.c_void_p
    w = ctypes.c_int.from_address(address())
    assert w.value == 0
    yield w
    w.value = 0


@pytest.fixture(scope="module")
def have(ft):
    g = synth.rng(31)
    sk = synth.scalars_mod_L(g, 1)[0]
    pk = ft.Array.from_scalars(sk[None]).to_bytes_folded()[0]
    m, r = synth.plaintexts(g, 40, 255), synth.scalars_mod_L(g, 40)
    a, b = ft.encrypt(pk, m, r, 8)
    return {"g": g, "sk": sk, "pk": pk, "m": m, "r": r, "a": a, "b": b, "enc": a.to_bytes_folded(),
            "long": ft.Array.from_scalars(synth.scalars_mod_L(g, 1 << 18)),
            "zero": ft.Array.init_scalar(40)}


WAITING = {
    "synchronize": lambda ft, h: ft.synchronize(),
    "to_bytes_folded": lambda ft, h: h["zero"].to_bytes_folded(),
    "to_bytes_affine": lambda ft, h: h["zero"].to_bytes_affine(),
    "to_bytes": lambda ft, h: h["zero"].to_bytes(),
    "to_packed": lambda ft, h: h["zero"].to_packed(),
    "from_bytes_folded": lambda ft, h: ft.Array.from_bytes_folded(h["enc"]),
    "validate": lambda ft, h: h["a"].validate(),
    "contains": lambda ft, h: h["a"].contains(h["b"]),
    "equal": lambda ft, h: h["a"].equal(h["b"]),
    "not_equal": lambda ft, h: h["a"].not_equal(h["b"]),
    "index": lambda ft, h: h["a"].index(),
    "reduce_isum": lambda ft, h: ft.Array.init_scalar(3).reduce_isum(np.arange(40) % 3, h["a"]),
    "encrypt": lambda ft, h: ft.encrypt(h["pk"], h["m"], h["r"], 8),
    "decrypt": lambda ft, h: ft.decrypt(h["a"], h["b"], h["sk"], 256),
}


@pytest.mark.parametrize("name", list(WAITING))
def test_set_while_a_call_waits(ft, have, word, name):
    WAITING[name](ft, have)  # (tables are built here)
    for _ in range(8):  # 40 ms of work that the call waits for
        have["long"].scale(have["sk"])
    timer = threading.Timer(0.01, lambda: setattr(word, "value", 1))
    timer.start()
    with pytest.raises(ft.FtError) as e:
        WAITING[name](ft, have)
    timer.join()
    assert e.value.code == INTERNAL and ft.api.lib().ftx_last_cuda_error() == TIMEOUT
    word.value = 0
    ft.synchronize()
    WAITING[name](ft, have)


ENTRY = {
    "init_scalar": lambda ft, h: ft.Array.init_scalar(3),
    "from_scalars": lambda ft, h: ft.Array.from_scalars(h["r"]),
    "add": lambda ft, h: h["zero"].add(h["a"]),
    "mul": lambda ft, h: h["zero"].mul(h["r"]),
    "scale": lambda ft, h: h["zero"].scale(h["sk"]),
    "neg": lambda ft, h: h["zero"].neg(),
    "scan": lambda ft, h: h["zero"].scan(),
    "rerandomise": lambda ft, h: ft.rerandomise(h["zero"], h["zero"], h["pk"], h["r"]),
    "server": lambda ft, h: ft.Server(h["pk"], 1 << 30, slots=2),
}


@pytest.mark.parametrize("name", list(ENTRY) + list(WAITING))
def test_set_before_a_call(ft, have, word, name):
    word.value = 1
    with pytest.raises(ft.FtError) as e:
        {**ENTRY, **WAITING}[name](ft, have)
    assert e.value.code == INTERNAL


def test_server_request(ft, have, word):
    """A request that runs when a kernel gives up ends with the error: its new
    arrays are nobody's, its bytes are back in the budget."""
    g, n = have["g"], 5000
    m, r = synth.plaintexts(g, n, 1), synth.scalars_mod_L(g, n)
    srv = ft.Server(have["pk"], 1 << 30, slots=2)
    c1, c2, _, _ = srv.wait(srv.submit_encrypt(m, r, 1))
    held = srv.stats()[0]
    off = synth.csr_offsets(g, n, 100)
    for submit in (lambda: srv.submit_encrypt(m, r, 1), lambda: srv.submit_rerand(c1, c2, r),
                   lambda: srv.submit_smul(c1, c2, r), lambda: srv.submit_segsum(c1, c2, off)):
        for _ in range(8):  # 40 ms of work that the request waits for
            have["long"].scale(have["sk"])
        ticket = submit()
        word.value = 1
        with pytest.raises(ft.FtError) as e:
            srv.wait(ticket)
        assert e.value.code == INTERNAL and srv.stats() == (held, 0, 0)
        word.value = 0
    d1, d2, _, _ = srv.wait(srv.submit_encrypt(m, r, 1))
    assert srv.stats()[0] == 2 * held
    srv.release(c1, c2, d1, d2)
    assert srv.stats() == (0, 0, 0)
    srv.close()
