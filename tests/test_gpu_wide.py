"""The one-warp decoder of wide order-1 alphabets, against the oracle.

Which decoder takes a wide alphabet depends on how many such streams a batch
holds, so a batch as small as a test's goes to the four-warp decoder; here
o1_four_max_streams 0 sends it to the one-warp decoder, and the stage
statistics say that it ran. Alphabets on both sides of every count of chains
per lane (20 / 21, 30 / 31, 40 / 41 contexts) and of the dense limit (47), data
that guesses well, badly, and badly only late in a stream, words at odd
addresses, streams cut off and with damaged words.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GROUP = 8 * 32
LENGTHS = [1, 31, 33, GROUP - 1, GROUP + 32, 9 * GROUP + 5, 200 * GROUP + 17]
# |D| counts context 0 as well: 16, 20, 21, 30, 31, 32, 33, 40, 41, 47
SYMBOLS = [15, 19, 20, 29, 30, 31, 32, 39, 40, 46]


def _symbols(rng, nsym):
    return np.sort(rng.choice(np.arange(1, 256), nsym, replace=False)).astype(np.uint8)


def _iid(rng, alphabet, n):
    p = 1.0 / np.arange(1, len(alphabet) + 1)
    return alphabet[rng.choice(len(alphabet), n, p=p / p.sum())]


def _cycle(rng, alphabet, n):
    step = np.where(rng.random(n) < 0.02, rng.integers(0, len(alphabet), n), 1)
    return alphabet[np.cumsum(step) % len(alphabet)]


def _late(rng, alphabet, n):
    """Long guessed stretches with a few wrong groups between them, the last
    of them near the end."""
    out = _iid(rng, alphabet, n)
    for at in (n // 3, n // 2, n - 2 * GROUP):
        if at > GROUP:
            out[at:at + GROUP] = _cycle(rng, alphabet, len(out[at:at + GROUP]))
    return out


def _spans(lens):
    lens = np.asarray(lens, np.uint64)
    return np.stack([np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint64), lens], 1)


@pytest.fixture
def wide_codec():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from fqxv_b200.batch import Codec

    c = Codec(0)
    c.set_param("o1_four_max_streams", 0)
    c.set_param("o1_top_max", 0)
    c.stage_stats(True)
    yield c
    c.close()


def _only_wide_ran(codec):
    st = codec.stage_stats(True)
    return st["dec_o1_wide"]["launches"] > 0 and st["dec_o1_dense"]["launches"] == 0


@pytest.mark.parametrize("nsym", SYMBOLS)
@pytest.mark.parametrize("make", [_iid, _cycle, _late])
def test_wide_streams_match_oracle(orc, wide_codec, nsym, make):
    import torch

    rng = np.random.default_rng(31 * nsym + len(make.__name__))
    alphabet = _symbols(rng, nsym)
    blocks = [make(rng, alphabet, n) for n in LENGTHS]
    for b in blocks:  # every symbol occurs in the streams long enough
        if len(b) > 4 * nsym:
            b[:nsym] = alphabet
    streams = [orc.encode(b.tobytes(), 1) for b in blocks]
    arena, spans = b"", []
    for i, s in enumerate(streams):  # odd and even addresses
        arena += b"\xff" * (1 + (len(arena) + i) % 2)
        spans.append([len(arena), len(s)])
        arena += s
    out_spans = _spans([len(b) for b in blocks])
    d_src = torch.from_numpy(np.frombuffer(arena, np.uint8).copy()).to("cuda")
    out, lens, status = wide_codec.decode_batch(d_src, np.array(spans, np.uint64), out_spans)
    assert _only_wide_ran(wide_codec)
    assert (status == 0).all() and (lens == out_spans[:, 1]).all()
    assert np.array_equal(out.cpu().numpy(), np.concatenate(blocks))


@pytest.mark.parametrize("nsym", [15, 30, 32, 46])
@pytest.mark.parametrize("make", [_iid, _cycle])
def test_damaged_wide_streams_end_as_the_oracles(orc, wide_codec, nsym, make):
    """Damaged words lead to symbols without a context, cut ones run out;
    status and bytes are the oracle's."""
    import torch

    rng = np.random.default_rng(5 * nsym + len(make.__name__))
    alphabet = _symbols(rng, nsym)
    streams = []
    for i, n in enumerate([40_001, 60_000, 60_000, 60_000, 50_000, 50_000]):
        block = make(rng, alphabet[:-1], n)
        block[-1] = alphabet[-1]  # the last symbol has no context of its own
        s = bytearray(orc.encode(block.tobytes(), 1))
        if i in (1, 2, 3):
            s[len(s) * (i + 5) // 9] ^= 0x55
        streams.append(bytes(s[:len(s) - 2 * 999] if i >= 4 else s))
    want = [orc.decode_status(s, max_len=1 << 16) for s in streams]
    assert want[0][0] == 0 and want[4][0] != 0
    out_spans = np.stack([np.arange(len(streams), dtype=np.uint64) << np.uint64(16),
                          np.full(len(streams), 1 << 16, np.uint64)], axis=1)
    d_src = torch.from_numpy(np.frombuffer(b"".join(streams), np.uint8).copy()).to("cuda")
    out, got, status = wide_codec.decode_batch(d_src, _spans([len(s) for s in streams]), out_spans, max_len=1 << 16,
                                               raise_on_error=False)
    assert _only_wide_ran(wide_codec)
    out = out.cpu().numpy()
    for i, (ws, wb) in enumerate(want):
        assert status[i] == ws, i
        if ws == 0:
            at = int(out_spans[i, 0])
            assert out[at:at + int(got[i])].tobytes() == wb, i
