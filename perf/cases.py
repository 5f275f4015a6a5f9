"""What the performance of this framework is measured on.

A case is one call, or one encode and decode pair, that a program makes through
the public entry points: the single-buffer calls (`rans.encode`, `rans.decode`),
the batched device API (`batch.Codec.encode_batch`, `decode_batch`), its
host-buffer forms, the block frames and the read-name tokenizer. The data have
the distributions of `fqxv_b200/workloads.py`, made on the GPU from the seed
alone: binned quality, full-range quality, ACGT, name tokens, ONT quality and
the quality random walk.

* `listed()`   the cases that are always measured.
* `draw(rng)`  one more case of the same ranges.
* `prepare`    what the program holds before the call (data, spans, a Codec).
* `run`        one pass; every output whole.
* `work`       the bytes a pass cannot avoid moving.
* `exact`      decoded bytes, known without any coder.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from fqxv_b200 import batch, rans, tokenizer

KiB, MiB = 1 << 10, 1 << 20
DEV = "cuda:0"
MIX = ("binned", "full", "acgt", "names")           # the mixed batch's stream types
KINDS = MIX + ("ont", "walk")
# Bits per symbol of each distribution at order 0 and order 1, for `work`.
BITS = {"binned": (0.97, 0.53), "full": (4.21, 3.89), "acgt": (2.01, 2.01), "names": (3.54, 3.22),
        "ont": (4.87, 4.76), "walk": (5.30, 2.67)}


def listed():
    return [
        # A single small buffer on the host, there and back: one name or
        # reorder sub-stream of a container block. Latency and launches.
        dict(name="call_16k", op="call", kind="names", size=16 * KiB, order=2),
        # One 1 MiB block of binned quality at order 0, there and back on the
        # device: a program that codes block by block.
        dict(name="block_1m_o0", op="roundtrip", kind="binned", blocks=1, lo=MiB, hi=MiB, order=0),
        # 64 blocks of 1 MiB of full-range quality at order 1: an archive
        # writer's, and a reader's, ordinary batch.
        dict(name="full_64_enc", op="encode", kind="full", blocks=64, lo=MiB, hi=MiB, order=1),
        dict(name="full_64_dec", op="decode", kind="full", blocks=64, lo=MiB, hi=MiB, order=1),
        # The mixed archive: 2048 blocks of 4 KiB to 4 MiB (odd lengths) of
        # four stream types, the smaller order kept. The largest work.
        dict(name="mixed_enc", op="encode", kind="mixed", blocks=2048, lo=4 * KiB, hi=4 * MiB, order=2),
        dict(name="mixed_dec", op="decode", kind="mixed", blocks=2048, lo=4 * KiB, hi=4 * MiB, order=2),
        # Many like-sized quality blocks of one order: a reader that streams a
        # whole lane of binned quality.
        dict(name="binned_512_dec_o0", op="decode", kind="binned", blocks=512, lo=512 * KiB, hi=512 * KiB, order=0),
        dict(name="binned_512_dec_o1", op="decode", kind="binned", blocks=512, lo=512 * KiB, hi=512 * KiB, order=1),
        # Long-read quality of one file: a few large ragged blocks at order 1.
        dict(name="ont_dec", op="decode", kind="ont", blocks=10, lo=256 * KiB, hi=8 * MiB, order=1),
        # A mixed batch between pinned host buffers, there and back.
        dict(name="mixed_host", op="host", kind="mixed", blocks=192, lo=4 * KiB, hi=4 * MiB, order=2),
        # Container frames: write, then walk and verify every CRC-32C.
        dict(name="frames", op="frames", kind="bytes", blocks=512, lo=4 * KiB, hi=4 * MiB, order=0),
        # Read names of 32 container blocks through the tokenizer and back.
        dict(name="names_32", op="names", kind="reads", blocks=32, lo=4000, hi=4000, order=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["call", "roundtrip", "encode", "encode", "decode", "decode", "decode", "host", "frames", "names"])
    order = rng.choice([0, 1, 2, 3])
    if op == "call":
        return dict(op=op, kind=rng.choice(KINDS), size=_log(rng, 64, 256 * KiB), order=order)
    if op == "names":
        return dict(op=op, kind="reads", blocks=_log(rng, 1, 32), lo=_log(rng, 100, 4000), hi=4000, order=2,
                    layout=rng.randrange(1 << 30))
    lo = _log(rng, 4 * KiB, MiB)
    hi = max(lo, _log(rng, 64 * KiB, 4 * MiB))
    # as many blocks as keep a case below 256 MiB (the largest listed: 1.2 GB)
    most = max(1, min(1024, 256 * MiB // hi))
    blocks = _log(rng, 1, most if op != "host" else max(1, most // 4))
    kind = "bytes" if op == "frames" else rng.choice(KINDS + ("mixed", "mixed"))
    return dict(op=op, kind=kind, blocks=blocks, lo=lo, hi=hi, order=0 if op == "frames" else order,
                layout=rng.randrange(1 << 30))


# ---- data -------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _binned(n, g, read_len=151):
    rows = -(-n // read_len)
    u = torch.rand((rows, read_len), generator=g, device=DEV)
    sym = torch.bucketize(u, torch.tensor([0.02, 0.07, 0.20], device=DEV)).to(torch.uint8)
    fresh = torch.rand((rows, read_len), generator=g, device=DEV) >= 0.7
    fresh[:, 0] = True
    at = torch.where(fresh, torch.arange(read_len, device=DEV, dtype=torch.int32), 0)
    sym = torch.gather(sym, 1, torch.cummax(at, 1).values.long())
    return torch.tensor(list(b"#,:F"), dtype=torch.uint8, device=DEV)[sym.long()].reshape(-1)[:n]


def _full(n, g, read_len=150):
    rows = -(-n // read_len)
    pos = torch.arange(read_len, device=DEV, dtype=torch.float32)
    q = torch.randn((rows, read_len), generator=g, device=DEV).mul_(3.0).add_(38.0 - 0.08 * pos).round_().clamp_(2, 41)
    tail = torch.rand((rows, 1), generator=g, device=DEV) < 0.01
    start = torch.randint(0, read_len, (rows, 1), generator=g, device=DEV)
    q[tail & (pos >= start)] = 2.0
    return (q.to(torch.uint8) + 33).reshape(-1)[:n]


def _acgt(n, g):
    out = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=DEV)[torch.randint(0, 4, (n,), generator=g, device=DEV)]
    out[torch.rand(n, generator=g, device=DEV) < 0.001] = ord("N")
    return out


def _decimal(v, width=7):
    a = v.abs()
    out = torch.zeros((len(v), width), dtype=torch.uint8, device=DEV)
    digits = torch.ones_like(a)
    t = a.clone()
    for col in range(width - 1, -1, -1):
        out[:, col] = (48 + t % 10).to(torch.uint8)
        t = t // 10
        digits += t > 0
    lead = (width - digits)[:, None]
    col = torch.arange(width, device=DEV)[None, :]
    out[col < lead] = 0
    out[(col == lead - 1) & (v < 0)[:, None]] = ord("-")
    return out


def _names(n, g):
    k = n // 12 + 16
    fields = [torch.randint(0, 65536, (k,), generator=g, device=DEV),
              torch.randint(0, 65536, (k,), generator=g, device=DEV),
              (torch.rand(k, generator=g, device=DEV) < 0.01).long(),
              torch.randint(0, 40, (k,), generator=g, device=DEV),
              torch.randint(-2000, 2000, (k,), generator=g, device=DEV)]
    cols = []
    for j, f in enumerate(fields):
        cols.append(_decimal(f))
        cols.append(torch.full((k, 1), ord(":") if j < 4 else ord("\n"), dtype=torch.uint8, device=DEV))
    text = torch.cat(cols, 1).reshape(-1)
    return text[text != 0][:n]


def _ont(n, g):
    reads = n // 4000 + 64
    while True:
        lens = (torch.randn(reads, generator=g, device=DEV) * 0.8 + math.log(8000.0)).exp_().long().clamp_(min=1)
        if int(lens.sum()) >= n:
            break
        reads *= 2
    means = torch.rand(reads, generator=g, device=DEV) * 15 + 10
    m = torch.repeat_interleave(means, lens)[:n]
    return (torch.randn(n, generator=g, device=DEV).mul_(6.0).add_(m).round_().clamp_(3, 40)).to(torch.uint8) + 33


def _walk(n, g, run=1024):
    rows = -(-n // run)
    step = torch.randint(-3, 4, (run, rows), generator=g, device=DEV, dtype=torch.int32)
    q = torch.full((rows,), 30, dtype=torch.int32, device=DEV)
    out = torch.empty((run, rows), dtype=torch.uint8, device=DEV)
    for i in range(run):
        q = (q + step[i]).clamp_(2, 41)
        out[i] = (q + 33).to(torch.uint8)
    return out.t().reshape(-1)[:n].contiguous()


def _bytes(n, g):
    return torch.randint(0, 256, (n,), generator=g, device=DEV, dtype=torch.uint8)


_GENERATORS = {"binned": _binned, "full": _full, "acgt": _acgt, "names": _names, "ont": _ont, "walk": _walk,
               "bytes": _bytes}


def _layout(case):
    """Block lengths (log-uniform in [lo, hi]) and the type of each block: the
    case's own, so that every seed fills the same shape."""
    nprng = np.random.default_rng(case.get("layout", 0))
    lo, hi = case["lo"], case["hi"]
    lens = np.exp(nprng.uniform(math.log(lo), math.log(hi), case["blocks"])).astype(np.int64).clip(lo, hi)
    kinds = nprng.integers(0, len(MIX), case["blocks"])
    spans = np.zeros((len(lens), 2), dtype=np.uint64)
    spans[1:, 0] = np.cumsum(lens)[:-1]
    spans[:, 1] = lens
    return spans, kinds


def _data(case, seed):
    """The input arena on the device and its block spans."""
    spans, kinds = _layout(case)
    total = int(spans[:, 1].sum())
    g = _gen(seed)
    if case["kind"] != "mixed":
        return _GENERATORS[case["kind"]](total, g), spans
    out = torch.empty(total, dtype=torch.uint8, device=DEV)
    for k, kind in enumerate(MIX):
        mine = spans[kinds == k]
        if not len(mine):
            continue
        pool, at = _GENERATORS[kind](int(mine[:, 1].sum()), g), 0
        for o, n in mine.astype(np.int64):
            out[o:o + n] = pool[at:at + n]
            at += n
    return out, spans


def _read_names(case, seed):
    """Illumina-style names, a list per block."""
    nprng = np.random.default_rng(seed)
    counts = np.random.default_rng(case.get("layout", 0)).integers(case["lo"], case["hi"] + 1, case["blocks"])
    out = []
    for b, k in enumerate(counts.tolist()):
        x, y = nprng.integers(1000, 32000, k), nprng.integers(1000, 32000, k)
        tile = 1101 + (np.arange(k) + int(nprng.integers(0, 400))) // 400
        tail = b" 1:N:0:ATCACG" if b % 2 else b""
        out.append([b"A00123:8:H7KJ2DSXX:%d:%d:%d:%d%s" % (1 + b % 4, t, i, j, tail)
                    for t, i, j in zip(tile.tolist(), x.tolist(), y.tolist())])
    return out


# ---- the program ------------------------------------------------------------

def _ends(spans):
    return int(spans[-1, 0] + spans[-1, 1])


def prepare(case, seed):
    op, s = case["op"], {"case": case}
    if op == "names":
        s["names"] = _read_names(case, seed)
        most = 64 * sum(len(b) for b in s["names"])
        s["enc"], s["out"] = np.zeros(most + 4096 * case["blocks"], dtype=np.uint8), np.zeros(most, dtype=np.uint8)
        return s
    if op == "call":
        s["src"] = _GENERATORS[case["kind"]](case["size"], _gen(seed)).cpu().numpy().tobytes()
        s["enc"] = np.zeros(rans.encode_bound(case["size"], case["order"]), dtype=np.uint8)
        return s
    data, spans = _data(case, seed)
    codec = s["codec"] = batch.Codec(0)
    s["spans"], n = spans, data.numel()
    if op == "frames":
        s["src"] = data
        s["dst"] = torch.zeros(codec.frame_bound(spans, True), dtype=torch.uint8, device=DEV)
    elif op == "host":
        s["src"] = torch.empty(n, dtype=torch.uint8, pin_memory=True)
        s["src"].copy_(data)
        s["enc"] = torch.zeros(codec.encode_bound(spans, case["order"]), dtype=torch.uint8, pin_memory=True)
        s["out"] = torch.empty(n, dtype=torch.uint8, pin_memory=True)
    else:
        if op != "decode":
            s["src"] = data
        s["enc"] = torch.zeros(codec.encode_bound(spans, case["order"]), dtype=torch.uint8, device=DEV)
        if op != "encode":
            s["out"] = torch.empty(n, dtype=torch.uint8, device=DEV)
        torch.cuda.synchronize()
        if op == "decode":
            # the streams as they came from a writer
            _, s["streams"], _ = codec.encode_batch(data, spans, case["order"], d_dst=s["enc"])
            s["enc"] = s["enc"][:_ends(s["streams"])].clone()
    torch.cuda.synchronize()
    return s


def _into(buf, data):
    """The bytes of a result, in the program's own buffer (zero behind them)."""
    buf[:len(data)] = np.frombuffer(data, dtype=np.uint8)
    return buf


def run(s):
    case = s["case"]
    op, order = case["op"], case.get("order", 0)
    if op == "call":
        enc = rans.encode(s["src"], rans.Order(order))
        dec = rans.decode(enc)
        return _into(s["enc"], enc), len(enc), np.frombuffer(dec, dtype=np.uint8)
    if op == "names":
        enc = tokenizer.encode_blocks(s["names"])
        dec = tokenizer.decode_blocks(enc)
        return (_into(s["enc"], b"".join(enc)), np.array([len(e) for e in enc]),
                _into(s["out"], b"\n".join(n for blk in dec for n in blk)))
    codec, spans = s["codec"], s["spans"]
    if op == "frames":
        framed, offs, crcs, total = codec.frame_blocks(s["src"], spans, terminate=True, d_dst=s["dst"])
        places, seen, status, consumed, ended = codec.read_blocks(framed, total)
        return framed, total, offs, crcs, places, seen, status, consumed, int(ended)
    if op == "host":
        streams, orders = codec.encode_batch_host(s["src"].numpy(), spans, order, s["enc"].numpy())
        lens, status = codec.decode_batch_host(s["enc"].numpy(), streams, spans, s["out"].numpy())
        return s["enc"], streams, orders, s["out"], lens, status
    if op == "encode":
        enc, streams, orders = codec.encode_batch(s["src"], spans, order, d_dst=s["enc"])
        return enc, streams, orders
    if op == "decode":
        out, lens, status = codec.decode_batch(s["enc"], s["streams"], spans, d_dst=s["out"])
        return out, lens, status
    enc, streams, orders = codec.encode_batch(s["src"], spans, order, d_dst=s["enc"])
    out, lens, status = codec.decode_batch(enc, streams, spans, d_dst=s["out"])
    return enc, streams, orders, out, lens, status


def work(case):
    """Bytes: an encode reads n and writes the streams, a decode the reverse;
    frames are read, written, and read again to be verified."""
    op = case["op"]
    if op == "names":
        n = case["blocks"] * (case["lo"] + case["hi"]) / 2 * 41.0
        return {"bytes": 2 * n * 1.2, "flops": 0.0}
    if op == "call":
        n = float(case["size"])
    else:
        lo, hi = case["lo"], case["hi"]
        n = case["blocks"] * (lo if hi == lo else (hi - lo) / math.log(hi / lo))
    if op == "frames":
        return {"bytes": 3.0 * n, "flops": 0.0}
    kinds = MIX if case["kind"] == "mixed" else (case["kind"],)
    order = case["order"]
    bits = sum(min(BITS[k]) if order >= 2 else BITS[k][order] for k in kinds) / len(kinds)
    one = n * (1.0 + bits / 8.0)
    return {"bytes": one * (1.0 if op in ("encode", "decode") else 2.0), "flops": 0.0}


def exact(case, seed):
    """Decoded bytes equal the input; coded bytes have no value of this kind."""
    op = case["op"]
    if op in ("names", "frames", "encode"):
        return None
    if op == "call":
        return None, None, _GENERATORS[case["kind"]](case["size"], _gen(seed)).cpu().numpy()
    data, spans = _data(case, seed)
    data, lens, status = data.cpu().numpy(), spans[:, 1].copy(), np.zeros(len(spans), dtype=np.int32)
    if op == "decode":
        return data, lens, status
    return None, None, None, data, lens, status
