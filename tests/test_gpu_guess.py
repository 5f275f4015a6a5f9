"""Order-1 decoders that guess contexts, against the oracle.

The one-warp decoders walk a fixed number of columns back from each position
and check the guessed contexts a group of eight rounds at a time
(csrc/rans_decode.cu). These streams sit where that can go wrong: alphabets on
both sides of the class boundaries (5 / 6 and 15 / 16 symbols with context 0),
data whose contexts never meet (a cycle: every guess wrong, so groups are
decoded again and the stream ends on the exact decoder), data that turns from
one kind to the other, lengths around a round and a group, and streams and
words at odd addresses.
"""

import numpy as np
import pytest

from fqxv_b200 import rans

pytestmark = pytest.mark.gpu

GROUP = 8 * 32
LENGTHS = [1, 31, 33, GROUP - 1, GROUP + 32, 9 * GROUP + 5, 200 * GROUP + 17]


def _symbols(rng, nsym):
    return np.sort(rng.choice(np.arange(1, 256), nsym, replace=False)).astype(np.uint8)


def _iid(rng, alphabet, n):
    p = 1.0 / np.arange(1, len(alphabet) + 1)
    return alphabet[rng.choice(len(alphabet), n, p=p / p.sum())]


def _cycle(rng, alphabet, n):
    """Mostly the next symbol in turn: a column permutes the contexts, so two
    chains that start apart stay apart."""
    step = np.where(rng.random(n) < 0.02, rng.integers(0, len(alphabet), n), 1)
    return alphabet[np.cumsum(step) % len(alphabet)]


def _turns(rng, alphabet, n):
    half = n // 2
    return np.concatenate([_iid(rng, alphabet, half), _cycle(rng, alphabet, n - half)])


@pytest.mark.parametrize("nsym", [1, 4, 5, 13, 14, 15, 31, 40])
@pytest.mark.parametrize("make", [_iid, _cycle, _turns])
def test_guessed_contexts_match_oracle(orc, nsym, make):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from fqxv_b200.batch import Codec

    rng = np.random.default_rng(7 * nsym + len(make.__name__))
    alphabet = _symbols(rng, nsym)
    blocks = [make(rng, alphabet, n) for n in LENGTHS]
    streams = [orc.encode(b.tobytes(), 1) for b in blocks]
    # one filler byte in front of every second stream: odd and even addresses
    arena, spans = b"", []
    for i, s in enumerate(streams):
        arena += b"\xff" * (1 + (len(arena) + i) % 2)
        spans.append([len(arena), len(s)])
        arena += s
    lens = np.array([len(b) for b in blocks], dtype=np.uint64)
    out_spans = np.stack([np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint64), lens], axis=1)
    d_src = torch.from_numpy(np.frombuffer(arena, dtype=np.uint8).copy()).to("cuda")
    want = np.concatenate(blocks)
    codec = Codec(0)
    try:
        for top_max in (0, 1000):  # with and without launch groups for the longest streams
            codec.set_param("o1_top_max", top_max)
            out, got, status = codec.decode_batch(d_src, spans, out_spans)
            assert (status == 0).all() and (got == lens).all()
            assert np.array_equal(out.cpu().numpy(), want)
    finally:
        codec.close()
    assert rans.decode(streams[-1]) == blocks[-1].tobytes()


@pytest.mark.parametrize("nsym", [31, 32, 33])
@pytest.mark.parametrize("zero", [False, True])
def test_first_context_need_not_be_a_symbol(orc, nsym, zero):
    """Context 0 takes an index behind the symbols' when byte 0 never occurs:
    around the 32 lanes of the four-warp decoder, good streams and streams with
    damaged words (which meet symbols that have no context) decode as the
    oracle's do."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from fqxv_b200.batch import Codec

    rng = np.random.default_rng(100 * nsym + zero)
    alphabet = _symbols(rng, nsym)
    if zero:
        alphabet[0] = 0
    streams = []
    for i, n in enumerate([1, 33, 5 * GROUP + 9, 40_001, 60_000, 60_000]):
        block = _iid(rng, alphabet[:-1], n)
        block[-1] = alphabet[-1]  # the last symbol has no context of its own
        s = bytearray(orc.encode(block.tobytes(), 1))
        if i >= 4:
            s[len(s) * 3 // 4] ^= 0x55
        streams.append(bytes(s))
    want = [orc.decode_status(s, max_len=1 << 16) for s in streams]
    lens = np.array([len(s) for s in streams], np.uint64)
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint64)
    out_offs = np.arange(len(streams), dtype=np.uint64) << np.uint64(16)
    out_spans = np.stack([out_offs, np.full(len(streams), 1 << 16, np.uint64)], axis=1)
    d_src = torch.from_numpy(np.frombuffer(b"".join(streams), np.uint8).copy()).to("cuda")
    codec = Codec(0)
    try:
        for top_max in (0, 1000):
            codec.set_param("o1_top_max", top_max)
            out, got, status = codec.decode_batch(d_src, np.stack([offs, lens], 1), out_spans, max_len=1 << 16,
                                                  raise_on_error=False)
            out = out.cpu().numpy()
            for i, (ws, wb) in enumerate(want):
                assert status[i] == ws, (top_max, i)
                if ws == 0:
                    assert out[int(out_offs[i]):int(out_offs[i]) + int(got[i])].tobytes() == wb, (top_max, i)
    finally:
        codec.close()


@pytest.mark.parametrize("per_sm", [1, 2, 3, 4])
@pytest.mark.parametrize("top_max", [5, 1000])
def test_top_groups_share_an_sm(orc, per_sm, top_max):
    """Small-alphabet top streams as warps of one CTA, a share of its shared
    memory each: more and fewer streams than warps, images from the smallest to
    the largest of the class, and like-sized streams that give up their groups."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from fqxv_b200.batch import Codec

    rng = np.random.default_rng(per_sm)
    sizes = [70_000 - 4_001 * i for i in range(7)]
    blocks = [_iid(rng, _symbols(rng, nsym), n) for nsym in (2, 5, 6, 13, 15, 31) for n in sizes]
    blocks += [_cycle(rng, _symbols(rng, 14), 70_000)]
    streams = [orc.encode(b.tobytes(), 1) for b in blocks]
    lens = np.array([len(s) for s in streams], np.uint64)
    spans = np.stack([np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint64), lens], 1)
    olens = np.array([len(b) for b in blocks], np.uint64)
    out_spans = np.stack([np.concatenate([[0], np.cumsum(olens)[:-1]]).astype(np.uint64), olens], 1)
    d_src = torch.from_numpy(np.frombuffer(b"".join(streams), np.uint8).copy()).to("cuda")
    codec = Codec(0)
    try:
        for name, v in (("o1_top_exclusive", 1), ("o1_top_latency_pct", 0), ("o1_top_max", top_max),
                        ("o1_top_small_per_sm", per_sm)):
            codec.set_param(name, v)
        out, _, status = codec.decode_batch(d_src, spans, out_spans)
        assert (status == 0).all()
        assert np.array_equal(out.cpu().numpy(), np.concatenate(blocks))
    finally:
        codec.close()
