"""The 2-D heat sweep's low regions: bands of 2 rows (4-row tiles, the smallest grids) and of 4 rows (16-row tiles),
sizes around their tiles and around the line between them, aligned and unaligned rows, launches short of
8 sweeps: bit-identical to the oracle; the ghost ring and the padding stay as they were."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,pitch,iters", [(3, 3, 8, 8), (111, 4, 113, 9), (112, 5, 116, 16), (224, 9, 226, 3), (225, 190, 228, 17),  # 4-row tiles
                                               (330, 330, 333, 8), (512, 512, 516, 18), (65, 3000, 68, 9), (448, 495, 450, 16), (1111, 65, 1116, 13)])
def test_low_bands(gb, torch_cuda, nx, ny, pitch, iters):
    torch = torch_cuda
    f = W.heat2d_padded(nx, ny, 1.0, nx * ny)
    f[-1, 1:] = 0.5
    f[1:, 0] = -0.25
    f[1:-1, -1] = 2.0
    host = np.full((ny + 2, pitch), 7.0, dtype=np.float32)
    host[:, : nx + 2] = f
    bufs = [torch.from_numpy(host).cuda(), torch.from_numpy(host).cuda()]
    ci = ctypes.c_int(-1)
    gb.call("appfis_gb_heat2d", bufs[0].data_ptr(), bufs[1].data_ptr(), nx, ny, pitch, iters, 0.2, 0.2, ctypes.byref(ci), None)
    gb.call("appfis_gb_stream_sync", None)
    want = host.copy()
    want[:, : nx + 2] = O.heat2d(f, iters, 0.2)
    assert ci.value == (-(-iters // 8)) % 2
    assert np.array_equal(bufs[ci.value].cpu().numpy(), want)
    other = bufs[1 - ci.value].cpu().numpy()
    other[1:-1, 1:nx + 1] = want[1:-1, 1:nx + 1]
    assert np.array_equal(other, want)
