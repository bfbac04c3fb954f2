"""The reductions' position arithmetic and float sums: boxes whose rows are shorter and longer than the
stride of all threads, one and many blocks, values that a float sum rounds, overflows or cannot hold;
and the one-launch periodic ghost refresh against the axis-by-axis definition."""
import ctypes
import math

import numpy as np
import pytest

from appfis_gb300 import workloads as W

pytestmark = pytest.mark.gpu
CODE = {np.dtype(np.float32): 0, np.dtype(np.float64): 1, np.dtype(np.int32): 2}


def _reduce(gb, torch, a, box, op, name="appfis_gb_reduce"):
    t = torch.from_numpy(a).cuda()
    out = torch.zeros(1, dtype=torch.int64 if a.dtype == np.int32 else torch.float64, device="cuda")
    gb.call(name, t.data_ptr(), CODE[a.dtype], a.shape[2], a.shape[1], (ctypes.c_int * 6)(*box), op, out.data_ptr(), None)
    gb.call("appfis_gb_stream_sync", None)
    return out.item()


# (nz, ny, nx) of the field and x0 x1 y0 y1 z0 z1: one element; one block (4096) and one more; rows of 1 and 2 elements;
# a row longer than every thread's stride; planes of one row; odd extents inside a padded field
@pytest.mark.parametrize("shape,box", [((1, 1, 1), (0, 1, 0, 1, 0, 1)), ((1, 64, 64), (0, 64, 0, 64, 0, 1)), ((1, 17, 241), (0, 241, 0, 17, 0, 1)),
                                       ((3, 5000, 3), (1, 2, 1, 4999, 1, 2)), ((2, 2000, 7), (2, 4, 0, 2000, 0, 2)),
                                       ((1, 2, 700001), (0, 700001, 0, 2, 0, 1)), ((400, 1, 301), (1, 300, 0, 1, 1, 399)),
                                       ((61, 130, 257), (1, 256, 1, 129, 1, 60))])
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int32])
def test_boxes(gb, torch_cuda, shape, box, dtype):
    n = int(np.prod(shape))
    u = W.uniform(n, n, -5, 5).reshape(shape)
    a = (u * 1e8).astype(dtype) if dtype == np.int32 else (u * np.exp(3 * u)).astype(dtype)
    v = a[box[4]:box[5], box[2]:box[3], box[0]:box[1]].reshape(-1)
    for name in ("appfis_gb_reduce", "appfis_gb_reduce_noalloc"):
        assert _reduce(gb, torch_cuda, a, box, 1, name) == v.min()
        if v.max() > 0:
            assert _reduce(gb, torch_cuda, a, box, 0, name) == v.max()
        s = _reduce(gb, torch_cuda, a, box, 2, name)
        if dtype == np.int32:
            assert s == int(v.astype(np.int64).sum())
        else:  # a double per element would be within one rounding per addition in the tree: 2^-53 x ~30 levels
            assert abs(s - math.fsum(v)) <= 2.0 ** -48 * math.fsum(np.abs(v))


@pytest.mark.parametrize("n", [5, 5000, 300001])
def test_float_sums_out_of_the_float_range(gb, torch_cuda, n):
    box = (0, n, 0, 1, 0, 1)
    a = np.full((1, 1, n), 3.0e38, dtype=np.float32)
    assert abs(_reduce(gb, torch_cuda, a, box, 2) / (float(a[0, 0, 0]) * n) - 1.0) < 1e-12
    a[0, 0, n // 2] = np.inf
    assert _reduce(gb, torch_cuda, a, box, 2) == math.inf
    a[0, 0, 1] = -np.inf
    assert math.isnan(_reduce(gb, torch_cuda, a, box, 2))
    a = np.full((1, 1, n), 1e-45, dtype=np.float32)
    assert _reduce(gb, torch_cuda, a, box, 2) == float(a[0, 0, 0]) * n
    a[0, 0, 0] = np.nan  # no comparison holds: NaN is passed over
    assert _reduce(gb, torch_cuda, a, box, 1) == float(a[0, 0, 1])
    # what a float sum would lose: one large value among small ones, and its opposite
    a = np.full((1, 1, n), 1.0, dtype=np.float32)
    a[0, 0, 0], a[0, 0, 3] = 1e20, -1e20
    big = n - 2 if n > 256 * 16 else None  # the two meet exactly only in different threads' double sums
    s = _reduce(gb, torch_cuda, a, box, 2)
    assert s == n - 2 or (big is None or abs(s - big) <= 2.0 ** -48 * 2e20)


@pytest.mark.parametrize("dims,ghost", [((3,), 1), ((70,), 5), ((12, 12), 4), ((41, 9), 3), ((5, 300), 1), ((9, 10, 11), 3), ((66, 3, 5), 1),
                                        ((131, 37, 29), 4), ((8, 8, 8), 2)])
@pytest.mark.parametrize("dtype", [np.uint8, np.float16, np.float32, np.float64])
def test_periodic_ghosts(gb, torch_cuda, dims, ghost, dtype):
    shape = tuple(reversed(dims))
    a = (W.uniform(7, int(np.prod(shape)), 0, 250)).reshape(shape).astype(dtype)
    want = a.copy()
    for axis in reversed(range(len(shape))):  # x, then y, then z, each over the full extent of the others
        v, d = np.moveaxis(want, axis, 0), shape[axis]
        v[:ghost] = v[d - 2 * ghost:d - ghost].copy()
        v[d - ghost:] = v[ghost:2 * ghost].copy()
    t = torch_cuda.from_numpy(a).cuda()
    gb.call("appfis_gb_ghost_periodic", t.data_ptr(), a.itemsize, len(dims), (ctypes.c_int * len(dims))(*dims), ghost, None)
    gb.call("appfis_gb_stream_sync", None)
    assert np.array_equal(t.cpu().numpy(), want)
