"""Runs of decode rounds without a check of the words left, on the CPU.

Inside a run the order-0 and one-warp order-1 decoders follow the word position
in 32 bits and take it back to 64 bits when the run ends
(csrc/rans_decode.cu), so a run's words have to stay below 2^32: beyond that the
position loses a multiple of 2^32, and a truncated stream reads as whole.
"""

import ctypes

import pytest

from fqxv_b200 import rans


def _fast_rounds(navail, wp, full, r):
    fn = rans.lib().fqxv_rans_test_fast_rounds
    fn.restype = ctypes.c_int64
    fn.argtypes = [ctypes.c_uint64] * 4
    return fn(navail, wp, full, r)


@pytest.mark.parametrize("navail,wp,full,r,want", [
    (0, 0, 10, 0, 0), (63, 0, 10, 0, 0), (95, 0, 10, 0, 0), (96, 0, 10, 0, 1), (96, 1, 10, 0, 0),
    (1000, 0, 10, 0, 10), (1000, 0, 10, 9, 1), (1000, 0, 10, 10, 0), (1000, 0, 10, 11, 0), (1000, 700, 10, 0, 7),
    (1000, 2000, 10, 0, 0)])
def test_runs_end_with_the_rounds_or_the_words(navail, wp, full, r, want):
    assert _fast_rounds(navail, wp, full, r) == want


@pytest.mark.parametrize("wp", [0, 1, (1 << 32) - 1, 1 << 32, (1 << 33) + 5, 1 << 40])
@pytest.mark.parametrize("words", [1 << 31, (1 << 32) - 32, 1 << 32, (1 << 32) + 64, (1 << 33) + 999, 1 << 42])
def test_position_survives_a_run_of_any_stream(wp, words):
    navail, full = wp + words + 64, words // 32
    cnt = _fast_rounds(navail, wp, full, 0)
    assert cnt > 0
    for taken in (0, 32 * cnt - 1, 32 * cnt):  # words that the run may take
        w32 = (wp + taken) & 0xFFFFFFFF
        back = wp + ((w32 - (wp & 0xFFFFFFFF)) & 0xFFFFFFFF)
        assert back == wp + taken
