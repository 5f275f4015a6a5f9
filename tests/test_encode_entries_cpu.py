"""The encode tables' exact division, on the CPU.

An encode entry gives v / f by one multiplication, without a correction step
(csrc/rans_common.cuh). Checked for every frequency against integer division
(crates/fqxv-rans/src/model.rs:125-133), at the states where a reciprocal that
is off shows first: the ends of every quotient's range, near zero, near
x_max = f << 20 and at random quotients between.
"""

import ctypes

import numpy as np

from fqxv_b200 import rans


def test_every_frequency_maps_exactly():
    fn = rans.lib().fqxv_rans_test_enc_map
    fn.argtypes = [ctypes.c_uint32, ctypes.c_uint32, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p]
    rng = np.random.default_rng(11)
    for f in range(1, 4097):
        cum = int(rng.integers(0, 4096 - f + 1))
        top = min(f << 20, 1 << 32)
        q = np.concatenate([np.arange(0, 4), top // f - 1 - np.arange(0, 4), rng.integers(0, top // f, 200)])
        v = np.concatenate([q * f, q * f + f - 1, q * f + f // 2])
        v = v[(v > 0) & (v < top)]
        want = ((v // f) * 4096 + v % f + cum) & 0xFFFFFFFF
        a, out = v.astype(np.uint32), np.zeros(len(v), dtype=np.uint32)
        assert fn(f, cum, a.ctypes.data, len(a), out.ctypes.data) == 0, f
        assert np.array_equal(out, want.astype(np.uint32)), f
