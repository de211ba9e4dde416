"""The identities behind the plain path's FP64 arithmetic (Fma64 in
csrc/mfc_device.cuh): a + b = fma(a, 1, b), a - b = fma(-b, 1, a) and
a * b = fma(a, b, -0.0), to the bit, signed zeros, subnormals, infinities
and rounding ties included.  The C library's fma rounds once, like the
GPU's; NaNs compare as NaN."""
import ctypes
import ctypes.util
import itertools
import struct

import numpy as np

_libm = ctypes.CDLL(ctypes.util.find_library("m") or "libm.so.6")
_libm.fma.restype = ctypes.c_double
_libm.fma.argtypes = [ctypes.c_double] * 3


def _bits(x: float) -> int:
    return 0 if x != x else struct.unpack("<Q", struct.pack("<d", x))[0] + 1


def _values():
    tiny, huge = np.finfo(np.float64).tiny, np.finfo(np.float64).max
    edge = [0.0, 5e-324, tiny, tiny * (1 - 2 ** -52), 1e-200, 1e-16, 0.5, 1.0, 1 + 2 ** -52, 1 - 2 ** -53, 1.5, 3.0,
            2.0 ** 53, 2.0 ** 53 + 2, 1e150, 1e200, huge, float("inf"), float("nan")]
    rng = np.random.default_rng(0)
    rand = (rng.uniform(1, 2, 40) * 2.0 ** rng.integers(-1070, 1000, 40)).tolist()
    near = rng.uniform(1, 2, 40).tolist()
    return [s * v for v in edge + rand + near for s in (1.0, -1.0)]


def test_sums_and_products_as_fused_operations_keep_every_bit():
    with np.errstate(all="ignore"):
        for a, b in itertools.product(_values(), repeat=2):
            x, y = np.float64(a), np.float64(b)
            assert _bits(_libm.fma(a, 1.0, b)) == _bits(float(x + y)), (a, b, "+")
            assert _bits(_libm.fma(-b, 1.0, a)) == _bits(float(x - y)), (a, b, "-")
            assert _bits(_libm.fma(a, b, -0.0)) == _bits(float(x * y)), (a, b, "*")
