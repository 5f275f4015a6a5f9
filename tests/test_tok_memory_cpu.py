"""What the tokenizer's Python front end reserves for a decode, on the CPU
(the host code over the C oracle's coder, as in test_tok_cpu.py): buffers of the
names' own size, whatever the payloads' is, and each payload decoded once."""

import ctypes
import os
import subprocess
import types

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture
def front(orc, monkeypatch):
    """fqxv_b200.tokenizer over the CPU library, with the bytes it asks numpy for."""
    from fqxv_b200 import rans, tokenizer

    lib = os.path.join(ROOT, "oracle", "_build", "libcallers_cpu.so")
    subprocess.check_call(["make", "-s", "-C", os.path.join(ROOT, "oracle"), lib])
    L = ctypes.CDLL(lib)
    product = rans.lib()
    for name in ("fqxv_tok_encode_host", "fqxv_tok_decode_host", "fqxv_tok_decode_host_alloc"):
        if hasattr(product, name):
            getattr(L, name).argtypes = getattr(product, name).argtypes
    L.fqxv_rans_status_message = product.fqxv_rans_status_message
    monkeypatch.setattr(rans, "lib", lambda: L)
    monkeypatch.setattr(tokenizer, "_codec", lambda device: types.SimpleNamespace(_h=1))
    asked = []

    def note(make):
        def f(shape, dtype=float, *a, **k):
            out = make(shape, dtype, *a, **k)
            asked.append(out.nbytes)
            return out
        return f

    for name in ("empty", "zeros"):
        monkeypatch.setattr(np, name, note(getattr(np, name)))
    return tokenizer, asked


def _blocks():
    rng = np.random.default_rng(3)
    return [[b"A00123:8:H7KJ2DSXX:%d:1101:%d:%d" % (b, x, y) for x, y in rng.integers(1000, 32000, (3000, 2))]
            for b in range(4)] + [[b"x" * 50] * 20_000, []]


def test_decode_reserves_what_the_names_take(front):
    tokenizer, asked = front
    blocks = _blocks()
    payloads = tokenizer.encode_blocks(blocks)
    asked.clear()
    assert tokenizer.decode_blocks(payloads) == blocks
    nnames, nbytes = sum(map(len, blocks)), sum(len(n) for b in blocks for n in b)
    assert sum(asked) <= nbytes + 16 * nnames + 4096


def test_failed_and_empty_blocks(front):
    tokenizer, asked = front
    payloads = tokenizer.encode_blocks([[b"a:1", b"a:2"], [b"", b""]])
    asked.clear()
    bad = payloads[0][:-3]
    names, status = tokenizer.decode_blocks([bad, payloads[1], payloads[0]], raise_on_error=False)
    assert names == [[], [b"", b""], [b"a:1", b"a:2"]] and status[0] != 0 and not status[1:].any()
    assert tokenizer.decode_blocks([]) == [] and sum(asked) < 4096
    with pytest.raises(Exception):
        tokenizer.decode_blocks([bad])


def test_a_buffer_that_cannot_be_had_is_an_error(front, monkeypatch):
    tokenizer, _ = front
    payloads = tokenizer.encode_blocks([[b"a:1"] * 1000])
    real = np.empty

    def refuse(shape, *a, **k):
        if np.prod(shape) >= 1000:
            raise MemoryError("no room")
        return real(shape, *a, **k)

    monkeypatch.setattr(np, "empty", refuse)
    with pytest.raises(MemoryError):
        tokenizer.decode_blocks(payloads)
    monkeypatch.setattr(np, "empty", real)
    assert tokenizer.decode_blocks(payloads) == [[b"a:1"] * 1000]
