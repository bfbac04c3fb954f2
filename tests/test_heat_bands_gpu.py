"""The time-blocked 2-D heat sweep over its tile heights (4, 8 and 12 warps by grid size), row alignments
(4, 2 and 1 elements), sizes around a tile's 112 columns and 16 / 48 / 80 rows, and counts that leave a
launch short of 8 sweeps: bit-identical to the oracle; ghost ring and padding stay as they were."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,pitch,lead,iters", [(1, 1, 3, 0, 9), (5, 300, 7, 0, 17), (110, 15, 112, 0, 8), (111, 16, 113, 0, 8), (112, 17, 116, 0, 7),
                                                    (113, 33, 116, 1, 16), (113, 33, 116, 2, 1), (223, 48, 228, 0, 15), (240, 100, 242, 0, 23),
                                                    (777, 900, 779, 0, 11), (776, 901, 780, 0, 10), (782, 863, 784, 0, 8), (1024, 1024, 1026, 0, 17),
                                                    (1007, 1041, 1012, 0, 9), (1300, 1210, 1302, 0, 3)])
def test_bands(gb, torch_cuda, nx, ny, pitch, lead, iters):
    torch = torch_cuda
    f = W.heat2d_padded(nx, ny, 1.0, nx + ny)
    f[-1, 1:] = 0.5  # every face counts
    f[1:, 0] = -0.25
    f[1:-1, -1] = 2.0
    host = np.full((ny + 2, pitch), 7.0, dtype=np.float32)
    host[:, : nx + 2] = f
    bufs = []
    for _ in range(2):
        flat = torch.zeros(lead + host.size, dtype=torch.float32, device="cuda")
        v = flat[lead:].view(host.shape)
        v.copy_(torch.from_numpy(host).cuda())
        bufs.append(v)
    ci = ctypes.c_int(-1)
    gb.call("appfis_gb_heat2d", bufs[0].data_ptr(), bufs[1].data_ptr(), nx, ny, pitch, iters, 0.2, 0.2, ctypes.byref(ci), None)
    gb.call("appfis_gb_stream_sync", None)
    want = host.copy()
    want[:, : nx + 2] = O.heat2d(f, iters, 0.2)
    assert ci.value == (-(-iters // 8)) % 2
    assert np.array_equal(bufs[ci.value].cpu().numpy(), want)
    other = bufs[1 - ci.value].cpu().numpy()  # the ghost ring and the padding of the other buffer
    other[1:-1, 1:nx + 1] = want[1:-1, 1:nx + 1]
    assert np.array_equal(other, want)
