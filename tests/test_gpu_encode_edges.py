"""Blocks that start and end where the encoder's chunk copies are cut.

The chunks of a block are copied in aligned granules of 16 bytes and none may
reach outside it (tests/test_encode_reads_cpu.py), so the lowest whole chunk of
a block at an unaligned address is read like the rounds below the chunks. Bytes
against the oracle, with and without the order-1 key array.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHUNK = 16 * 32


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("keys", [0, 1])
def test_chunk_edges_match_oracle(orc, order, keys):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from fqxv_b200.batch import Codec

    rng = np.random.default_rng(2 * order + keys)
    p = 1.0 / np.arange(1, 36)
    spans, at = [], 0
    for off in (0, 1, 7, 8, 15):
        for n in (CHUNK - 32, CHUNK, CHUNK + 1, 2 * CHUNK, 2 * CHUNK + 31, 3 * CHUNK + 32, 9 * CHUNK, 9 * CHUNK + 5):
            at += (off - at) % 16
            spans.append([at, n])
            at += n
    data = (33 + rng.choice(len(p), at, p=p / p.sum())).astype(np.uint8)
    codec = Codec(0)
    try:
        codec.set_param("enc_o1_keys", keys)
        d_src = torch.from_numpy(data).to("cuda")
        out, osp, _ = codec.encode_batch(d_src, np.array(spans, np.uint64), order)
        out = out.cpu().numpy()
    finally:
        codec.close()
    for (o, n), (e, m) in zip(spans, osp.astype(np.int64)):
        assert out[e:e + m].tobytes() == orc.encode(data[o:o + n].tobytes(), order), (o % 16, n)
