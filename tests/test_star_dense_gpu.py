"""The radius-4 star on rows that are not 16-byte aligned, on grids that take the asynchronous-copy tile: bit
for bit the oracle's reference form and the scalar tile's weighted and FP16 results, for every word
size of the copies, ragged tiles and z chunks; padding and halo stay as they were."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu
AUTO, SCALAR2 = 0, 2


def _run(gb, torch, host, dtype, nx, ny, nz, pitch, lead, iters, mode, tile, kz):
    bufs = []
    for _ in range(2):
        flat = torch.zeros(lead + host.size, dtype=dtype, device="cuda")
        v = flat[lead:].view(host.shape)
        v.copy_(torch.from_numpy(host).cuda())
        bufs.append(v)
    w = (ctypes.c_float * 5)(*W.fdtd_weights()) if mode == 1 else None
    ci = ctypes.c_int(-1)
    gb.call("appfis_gb_star_r4", bufs[0].data_ptr(), bufs[1].data_ptr(), 0 if dtype == torch.float32 else 3, nx, ny, nz, pitch, iters, mode, 0.1, w,
            tile, kz, ctypes.byref(ci), None)
    gb.call("appfis_gb_stream_sync", None)
    return bufs[ci.value].float().cpu().numpy()


# FP32: 8-byte words (even pitch), 4-byte words (odd pitch; a pitch of a multiple of 4 one element off its
# alignment); FP16: 8-byte words (pitch 4 mod 8), 4-byte words (pitch 2 mod 4); tiles cut in x and y
@pytest.mark.parametrize("dtype,nx,ny,nz,pitch,lead,kz", [("f32", 130, 141, 150, 138, 0, 0), ("f32", 129, 160, 101, 138, 0, 5), ("f32", 64, 177, 181, 74, 0, 64),
                                                          ("f32", 255, 131, 125, 263, 0, 0), ("f32", 257, 129, 122, 268, 1, 9),
                                                          ("f16", 132, 141, 120, 140, 0, 0), ("f16", 186, 120, 99, 194, 0, 7), ("f16", 187, 121, 99, 196, 0, 0)])
def test_large_dense(gb, torch_cuda, dtype, nx, ny, nz, pitch, lead, kz):
    torch = torch_cuda
    td = torch.float32 if dtype == "f32" else torch.float16
    f = W.fdtd_padded(nx, ny, nz, nx + ny)
    f[:4] = 0.25  # a halo that counts
    f[:, :, -4:] = -0.5
    host = np.full(f.shape[:2] + (pitch,), 3.0, dtype=np.float32)
    host[..., : nx + 8] = f
    for mode in (0, 1):
        got = _run(gb, torch, host, td, nx, ny, nz, pitch, lead, 3, mode, AUTO, kz)
        want = _run(gb, torch, host, td, nx, ny, nz, pitch, lead, 3, mode, SCALAR2, 0)
        assert np.array_equal(got, want)
        assert (got[..., nx + 8:] == 3.0).all()
        if dtype == "f32" and mode == 0:
            assert np.array_equal(got[..., : nx + 8], O.star_r4(f, 3, coeff=0.1))
