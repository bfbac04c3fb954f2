"""FP32 SUM at every size as accurate as one addition to a double per element: values of a wide range that repeat
with the stride of all threads, so that every thread makes the same error and none cancels another; large values that meet
their opposites; sums that leave the float range."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 16 positive floats each (bit patterns) over 6 and 9 decades, on which a sum in two floats is off by 2^-45.7 and 2^-44.8
PATTERNS = [[0x40c082bc, 0x38640063, 0x3f02b13f, 0x398febf9, 0x3f639d9b, 0x4904b131, 0x3f17739f, 0x3b87425a,
             0x39a1d5a7, 0x3f932b50, 0x3cb03dbd, 0x426b9231, 0x3d70bde1, 0x3d9363bb, 0x3ec58740, 0x3c82f339],
            [0x40f84cfb, 0x3888d193, 0x3f0b203a, 0x3c19ade6, 0x412d19b4, 0x488195ab, 0x413cb549, 0x440fbed3,
             0x405e31e8, 0x3c2e7429, 0x3f23308c, 0x3a910329, 0x420d40c2, 0x431589c4, 0x4464f1fe, 0x3c8ce5c9]]


def _sum(gb, torch, a):
    t = torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    n = t.numel()
    gb.call("appfis_gb_reduce", t.data_ptr(), 0, n, 1, (ctypes.c_int * 6)(0, n, 0, 1, 0, 1), 2, out.data_ptr(), None)
    gb.call("appfis_gb_stream_sync", None)
    return out.item()


def _stride(torch, n):
    """Elements between one that a thread takes and its next: 16 elements a thread, at most 4 blocks of 256 threads per SM."""
    blocks = 1 if n <= 4096 else min(-(-n // 4096), 4 * torch.cuda.get_device_properties(0).multi_processor_count)
    return 256 * blocks


@pytest.mark.parametrize("n", [4096, 1 << 16, 1 << 20, 1 << 21])
@pytest.mark.parametrize("pattern", PATTERNS)
def test_values_that_repeat_with_the_stride(gb, torch_cuda, pattern, n):
    p = np.array(pattern, dtype=np.uint32).view(np.float32)
    a = np.repeat(p, _stride(torch_cuda, n))
    assert a.size == n
    # every thread has the same 16 values: its sum in doubles is off by 15 roundings at most, and the tree over threads
    # doubles equal values, exactly
    exact = math.fsum(p) * (n // 16)
    assert abs(_sum(gb, torch_cuda, a) - exact) <= 15 * 2.0 ** -53 * exact


@pytest.mark.parametrize("n", [5000, 300001, (1 << 20) + 3, 3000001])
def test_opposite_values_leave_the_small_ones(gb, torch_cuda, n):
    s = _stride(torch_cuda, n)
    for big, first, second in ((1e10, 0, 3), (1e10, 5, 5 + s), (1e20, 7, 7 + s), (1e20, 1, 1 + 3 * s)):  # 1e10: a double holds the sum exactly
        a = np.ones(n, dtype=np.float32)
        a[first], a[second] = big, -big
        assert _sum(gb, torch_cuda, a) == n - 2, (big, first, second)


@pytest.mark.parametrize("n", [(1 << 20) + 3, 3000001])
def test_large_boxes_out_of_the_float_range(gb, torch_cuda, n):
    a = np.full(n, 3.0e38, dtype=np.float32)
    assert abs(_sum(gb, torch_cuda, a) / (float(a[0]) * n) - 1.0) < 1e-12
    a[n // 2] = np.inf
    assert _sum(gb, torch_cuda, a) == math.inf
    a[1] = -np.inf
    assert math.isnan(_sum(gb, torch_cuda, a))
    a = np.full(n, 1e-45, dtype=np.float32)
    assert _sum(gb, torch_cuda, a) == float(a[0]) * n
