"""Read-name tokenizer over the B200 coder, shaped like
`crates/fqxv-tokenizer/src/lib.rs`:

    encode(names) -> bytes          lib.rs:482
    decode(src) -> list[bytes]      lib.rs:543

plus the batched forms `encode_blocks` / `decode_blocks`, which code every
role stream of every block in one GPU pass (libfqxv_rans_gpu.so,
`fqxv_tok_encode_host` / `fqxv_tok_decode_host`). Payloads are byte-identical
to the reference's. Errors: `Malformed` with the reference's
"malformed name stream: ..." text, or `rans.Malformed` for a role stream's
rANS error. There is no CPU fallback.
"""

from __future__ import annotations

import ctypes

import numpy as np

from . import rans

TOK_STATUSES = set(range(48, 62))


class Malformed(rans.Error):
    """lib.rs:40-50 Error::Malformed."""


def _raise(status: int) -> None:
    if status in TOK_STATUSES:
        raise Malformed(status, rans.status_message(status))
    rans.raise_for(status)


def _codec(device: int):
    from . import frame

    return frame.codec(device)


def _spans(lens) -> np.ndarray:
    """(offset, length) of items laid back to back; lens: any sized iterable
    of ints."""
    out = np.zeros((len(lens), 2), dtype=np.uint64)
    out[:, 1] = lens if isinstance(lens, np.ndarray) else np.fromiter(lens, dtype=np.uint64, count=len(lens))
    if len(out):
        np.cumsum(out[:-1, 1], out=out[1:, 0])
    return out


def _lens(items) -> np.ndarray:
    return np.fromiter(map(len, items), dtype=np.uint64, count=len(items))


def encode_blocks(blocks, device: int = 0) -> list[bytes]:
    """One payload per block of names (each a list of bytes-like names)."""
    names = [n if type(n) is bytes else bytes(n) for blk in blocks for n in blk]
    arena = np.frombuffer(b"".join(names) or b"\0", dtype=np.uint8)
    nsp = _spans(_lens(names))
    counts = [len(blk) for blk in blocks]
    bsp = _spans(counts)
    c = _codec(device)
    L = rans.lib()
    out = np.zeros((max(len(blocks), 1), 2), dtype=np.uint64)
    need = ctypes.c_uint64(0)
    cap = 4 * arena.size + 4096 * len(blocks) + (1 << 16)
    for _ in range(2):
        dst = np.empty(max(cap, 1), dtype=np.uint8)
        st = L.fqxv_tok_encode_host(c._h, arena.ctypes.data, nsp.ctypes.data, len(names), bsp.ctypes.data,
                                    len(blocks), dst.ctypes.data, dst.size, out.ctypes.data, ctypes.byref(need))
        if st == 17 and need.value > cap:
            cap = need.value
            continue
        _raise(st)
        return [dst[int(o):int(o + n)].tobytes() for o, n in out[:len(blocks)]]
    _raise(17)


def decode_blocks(payloads, device: int = 0, raise_on_error: bool = True):
    """Names of each payload; with raise_on_error False, (names per block,
    statuses) with an empty list for a failed block."""
    payloads = [bytes(p) for p in payloads]
    arena = np.frombuffer(b"".join(payloads) or b"\0", dtype=np.uint8)
    psp = _spans(_lens(payloads))
    n = len(payloads)
    c = _codec(device)
    L = rans.lib()
    blocks = np.zeros((max(n, 1), 2), dtype=np.uint64)
    status = np.zeros(max(n, 1), dtype=np.int32)
    bufs, failed = [], []

    def alloc(_, nbytes, nnames, names_p, spans_p):
        try:
            bufs[:] = np.empty(nbytes, dtype=np.uint8), np.empty((nnames, 2), dtype=np.uint64)
        except BaseException as e:
            failed.append(e)
            return 1
        names_p[0], spans_p[0] = (a.ctypes.data for a in bufs)
        return 0

    st = L.fqxv_tok_decode_host_alloc(c._h, arena.ctypes.data, psp.ctypes.data, n, rans.TokAlloc(alloc), None,
                                      blocks.ctypes.data, status.ctypes.data)
    if failed:
        raise failed[0]
    if st and st not in TOK_STATUSES and st not in rans.MALFORMED:
        _raise(st)
    # One bytes object, sliced by plain ints: a numpy slice and copy per name
    # took most of a call (128,000 names).
    h_names, nsp = bufs
    text = h_names.tobytes()
    out = []
    for b in range(n):
        f, k = int(blocks[b, 0]), int(blocks[b, 1])
        at = nsp[f:f + k, 0]
        out.append([text[i:j] for i, j in zip(at.tolist(), (at + nsp[f:f + k, 1]).tolist())])
    if raise_on_error:
        for s in status[:n]:
            if s:
                _raise(int(s))
        return out
    return out, status[:n].copy()


def encode(names, device: int = 0) -> bytes:
    """lib.rs:482 `encode(names)`."""
    return encode_blocks([list(names)], device)[0]


def decode(src, device: int = 0) -> list[bytes]:
    """lib.rs:543 `decode(src)`."""
    return decode_blocks([src], device)[0]
