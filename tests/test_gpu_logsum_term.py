"""The term of rc_logsum (recheck.c:260-265) that the device Forward runs, log1pf(expf(-t)) as one
function for 0 <= t <= 50, against the host libm's two calls: the same bits at every fifth float of
the range, and at every float of the stretches where the evaluation changes its path (t at 0 and
among the subnormals, expf(-t) around 0.41422, where log1pf's reduction starts, and around 2^-29,
and t up to 50)."""
import ctypes as C
import os
import struct

import numpy as np
import pytest

from protlocus_b200 import lib as L

pytestmark = pytest.mark.gpu

LIB = os.path.join(os.path.dirname(__file__), "..", "oracle", "_build", "liblmcheck.so")


def _bits(f):
    return struct.unpack("<I", struct.pack("<f", f))[0]


@pytest.mark.parametrize("lo,hi,stride", [
    (0, _bits(50.0) + 1, 5), (0, 1 << 20, 1), ((1 << 23) - (1 << 18), (1 << 23) + (1 << 18), 1),
    (_bits(0.8812), _bits(0.8816), 1), (_bits(20.09), _bits(20.12), 1), (_bits(49.9), _bits(50.0) + 1, 1)])
def test_term_equals_host(lo, hi, stride):
    if not os.path.exists(LIB):
        pytest.skip("oracle/_build/liblmcheck.so not built")
    host, lib = C.CDLL(LIB), L.load()
    host.lm_host.argtypes = [C.c_int, C.c_uint32, C.c_uint32, C.c_int64, C.c_void_p]
    total = -(-(hi - lo) // stride)
    chunk = 1 << 26
    dev, ref = np.empty(chunk, np.float32), np.empty(chunk, np.float32)
    for at in range(0, total, chunk):
        n, start = min(chunk, total - at), lo + at * stride
        assert lib.pl_rc_mathf_eval(0, 6, start, stride, n, dev.ctypes.data) == 1
        host.lm_host(6, start, stride, n, ref.ctypes.data)
        bad = dev[:n].view(np.uint32) != ref[:n].view(np.uint32)
        assert not bad.any(), hex(start + stride * int(np.argmax(bad)))
