"""The heat sweep's tallest region (12 warps of 8 rows, taken where every SM has one tile at most) at every alignment
of rows and fields (4, 2 and 1 elements), edges inside and at a tile's end: bit-identical to the oracle, ghost ring
and padding as they were."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pitch,lead", [(0, 0), (1, 0), (2, 0), (3, 0), (2, 1), (2, 2)])
@pytest.mark.parametrize("nx,ny,iters", [(1024, 1024, 9), (1006, 1120, 16), (1119, 1040, 3)])
def test_alignments(gb, torch_cuda, nx, ny, iters, pitch, lead):
    torch = torch_cuda
    pitch = (nx + 2 + 3) // 4 * 4 + pitch
    f = W.heat2d_padded(nx, ny, 1.0, nx + ny)
    f[-1, 1:] = 0.5
    f[1:, 0] = -0.25
    f[1:-1, -1] = 2.0
    host = np.full((ny + 2, pitch), 7.0, dtype=np.float32)
    host[:, :nx + 2] = f
    bufs = []
    for _ in range(2):
        flat = torch.zeros(lead + host.size, dtype=torch.float32, device="cuda")
        v = flat[lead:].view(host.shape)
        v.copy_(torch.from_numpy(host).cuda())
        bufs.append(v)
    torch.cuda.synchronize()
    ci = ctypes.c_int(-1)
    gb.call("appfis_gb_heat2d", bufs[0].data_ptr(), bufs[1].data_ptr(), nx, ny, pitch, iters, 0.2, 0.2, ctypes.byref(ci), None)
    gb.call("appfis_gb_stream_sync", None)
    want = host.copy()
    want[:, :nx + 2] = O.heat2d(f, iters, 0.2)
    assert np.array_equal(bufs[ci.value].cpu().numpy(), want)
