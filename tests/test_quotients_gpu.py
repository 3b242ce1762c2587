"""Quotients formed from a reciprocal (quotientBy, the final value of plain,
guided and mean sums; downRangeWeight, Downsample's range weight of integer
samples) equal the division bit for bit on the device: 2^30 seeded FP64 pairs
over the range of the sums, and every float of the weight's range."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import lgcr


def test_quotients_equal_the_division():
    fn = lgcr.library().lgcr_selftest_quotients
    fn.argtypes = [ctypes.POINTER(ctypes.c_uint64)]
    fn.restype = ctypes.c_int
    bad = (ctypes.c_uint64 * 2)(1, 1)
    assert fn(bad) == 0, lgcr.library().lgcr_last_error()
    assert list(bad) == [0, 0]
