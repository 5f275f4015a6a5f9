"""What the encoder's chunk copies read, on the CPU.

They go in aligned granules of 16 bytes, and a block starts and ends anywhere,
but no byte outside the block is read (csrc/rans_common.cuh, SymbolPlan).
"""

import ctypes

import pytest

from fqxv_b200 import rans

CHUNK = 16 * 32


def _reads(first, n, size):
    fn = rans.lib().fqxv_rans_test_enc_reads
    fn.restype = None
    fn.argtypes = [ctypes.c_uint64, ctypes.c_uint64, ctypes.c_uint32, ctypes.c_void_p, ctypes.c_void_p]
    lo, hi = ctypes.c_uint64(0), ctypes.c_uint64(0)
    fn(first, n, size, ctypes.byref(lo), ctypes.byref(hi))
    return lo.value, hi.value


@pytest.mark.parametrize("size", [1, 2])
@pytest.mark.parametrize("chunks", [0, 1, 2, 9])
def test_chunk_copies_stay_inside_the_block(size, chunks):
    for off in range(0, 32, size):
        first = (1 << 30) + off
        for rest in (0, 1, 2, 3, 7, 8, 15, 16, 31, 32, 33, 47, 64, 15 * 32, CHUNK - 1):
            n = chunks * CHUNK + rest
            lo, hi = _reads(first, n, size)
            assert first <= lo <= hi <= first + n * size, (off, rest)
            # every whole chunk but the lowest is copied, to the last round
            full_end = first + n // 32 * 32 * size
            if hi > lo:
                assert hi >= full_end and lo - first < 2 * CHUNK * size, (off, rest)
            else:
                assert n < 2 * CHUNK, (off, rest)
