"""Which decoder a batch's wide order-1 alphabets go to, from the stage
statistics; bytes against the input either way."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _decoders(codec, nwide, nother, n):
    """Launches of the four-warp and of the one-warp decoder for a batch of
    like-sized order-1 blocks, `nwide` of them of a wide alphabet."""
    import torch

    rng = np.random.default_rng(nwide + nother)
    wide = 40 + rng.integers(0, 30, (nwide, n))
    other = 40 + rng.integers(0, 4, (nother, n))
    data = np.concatenate([wide, other]).astype(np.uint8).reshape(-1)
    lens = np.full(nwide + nother, n, np.uint64)
    spans = np.stack([np.arange(len(lens), dtype=np.uint64) * np.uint64(n), lens], 1)
    d_src = torch.from_numpy(data).to("cuda")
    enc, streams, _ = codec.encode_batch(d_src, spans, 1)
    codec.stage_stats(True)
    out, _, status = codec.decode_batch(enc, streams, spans)
    st = codec.stage_stats(True)
    assert (status == 0).all() and torch.equal(out[:len(data)], d_src)
    return st["dec_o1_dense"]["launches"], st["dec_o1_wide"]["launches"]


@pytest.fixture
def codec():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from fqxv_b200.batch import Codec

    c = Codec(0)
    yield c
    c.close()


@pytest.mark.parametrize("value,four", [(0, False), (6, False), (7, True), (1 << 30, True)])
def test_parameter_counts_the_streams_of_a_launch_group(codec, value, four):
    codec.set_param("o1_four_max_streams", value)
    codec.set_param("o1_top_max", 0)
    assert _decoders(codec, 6, 20, 5000) == ((1, 0) if four else (0, 1))


@pytest.mark.parametrize("wide,others,four", [(1, 0, True), (444, 0, True), (445, 0, False), (120, 500, True),
                                              (440, 200, False)])
def test_rule_counts_wide_streams_and_a_share_of_the_others(codec, wide, others, four):
    if codec.get_param("o1_four_max_streams") != -1:
        codec.set_param("o1_four_max_streams", -1)
    codec.set_param("o1_top_max", 0)
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms != 148:
        pytest.skip("sizes are for 148 SMs")
    assert _decoders(codec, wide, others, 700) == ((1, 0) if four else (0, 1))


def test_long_wide_streams_beside_many_short_ones(codec):
    """More like-sized longest streams than a top group holds, and more short
    ones than the four-warp decoder takes: the longest go there alone."""
    import torch

    rng = np.random.default_rng(1)
    lens = np.array([200_000] * 12 + [1000] * 500, np.uint64)
    spans = np.stack([np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint64), lens], 1)
    data = (40 + rng.integers(0, 30, int(lens.sum()))).astype(np.uint8)
    d_src = torch.from_numpy(data).to("cuda")
    codec.set_param("o1_four_max_streams", -1)
    codec.set_param("o1_top_max", 4)
    enc, streams, _ = codec.encode_batch(d_src, spans, 1)
    codec.stage_stats(True)
    out, _, status = codec.decode_batch(enc, streams, spans)
    st = codec.stage_stats(True)
    assert (status == 0).all() and torch.equal(out[:len(data)], d_src)
    assert st["dec_o1_dense"]["launches"] == 1 and st["dec_o1_wide"]["launches"] == 1


@pytest.mark.parametrize("exclusive,want", [(1, (1, 1)), (0, (2, 0))])
def test_rule_leaves_out_the_sms_of_top_streams(codec, exclusive, want):
    """100 top streams on SMs of their own leave room for fewer than the 150
    others on the four-warp decoder; without SMs of their own all 250 fit."""
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes are for 148 SMs")
    rng = np.random.default_rng(2)
    lens = np.array([60_000] * 100 + [3000] * 150, np.uint64)
    spans = np.stack([np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint64), lens], 1)
    data = (40 + rng.integers(0, 30, int(lens.sum()))).astype(np.uint8)
    d_src = torch.from_numpy(data).to("cuda")
    for name, v in (("o1_four_max_streams", -1), ("o1_top_max", 111), ("o1_top_latency_pct", 75),
                    ("o1_top_exclusive", exclusive)):
        codec.set_param(name, v)
    enc, streams, _ = codec.encode_batch(d_src, spans, 1)
    codec.stage_stats(True)
    out, _, status = codec.decode_batch(enc, streams, spans)
    st = codec.stage_stats(True)
    assert (status == 0).all() and torch.equal(out[:len(data)], d_src)
    assert (st["dec_o1_dense"]["launches"], st["dec_o1_wide"]["launches"]) == want
