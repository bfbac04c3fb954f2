"""The radius-4 star's default tile on rows that are not 16-byte aligned, where the grid is a few planes thin or
its columns fill 64-wide tiles badly: as fast as the scalar tile, and its results bit for bit, on both sides of each line."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import workloads as W

pytestmark = pytest.mark.gpu
AUTO, SCALAR2 = 0, 2


def _run(gb, torch, a, b, dims, pitch, mode, tile, iters=2):
    w = (ctypes.c_float * 5)(*W.fdtd_weights())
    ci = ctypes.c_int(-1)
    stream = torch.cuda.current_stream()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    gb.call("appfis_gb_star_r4", a.data_ptr(), b.data_ptr(), 0 if a.dtype == torch.float32 else 3, *dims, pitch, iters, mode, 0.1, w, tile, 0,
            ctypes.byref(ci), stream.cuda_stream)
    e1.record()
    torch.cuda.synchronize()
    return (a if ci.value == 0 else b), e0.elapsed_time(e1)


# odd pitch (4-byte words): 15 and 16 planes, 96 and 97 columns; even: 7 and 8 planes; FP16: 1 and 2
@pytest.mark.parametrize("dtype,nx,ny,nz,pitch", [("f32", 601, 450, 15, 609), ("f32", 601, 450, 16, 609), ("f32", 96, 300, 140, 105),
                                                  ("f32", 97, 300, 140, 105), ("f32", 600, 500, 7, 610), ("f32", 600, 500, 8, 610),
                                                  ("f32", 2001, 2003, 1, 2009), ("f16", 1502, 1400, 1, 1510), ("f16", 1502, 700, 2, 1510)])
@pytest.mark.parametrize("mode", [0, 1])
def test_both_sides(gb, torch_cuda, dtype, nx, ny, nz, pitch, mode):
    torch = torch_cuda
    td = torch.float32 if dtype == "f32" else torch.float16
    host = np.full((nz + 8, ny + 8, pitch), 3.0, dtype=np.float32)
    host[..., :nx + 8] = W.uniform(nx, (nz + 8) * (ny + 8) * (nx + 8), -1, 1).reshape(nz + 8, ny + 8, nx + 8)
    src = torch.from_numpy(host).cuda().to(td)
    got, _ = _run(gb, torch, src.clone(), src.clone(), (nx, ny, nz), pitch, mode, AUTO)
    want, _ = _run(gb, torch, src.clone(), src.clone(), (nx, ny, nz), pitch, mode, SCALAR2)
    assert torch.equal(got, want)
    assert not torch.equal(got, src)


@pytest.mark.parametrize("nx,ny,nz,pitch", [(3000, 3000, 1, 3009), (3000, 3000, 1, 3010), (3000, 3000, 2, 3009), (3000, 3000, 2, 3010)])
def test_thin_grids_are_no_slower(gb, torch_cuda, nx, ny, nz, pitch):
    torch = torch_cuda
    a = torch.zeros((nz + 8, ny + 8, pitch), device="cuda")
    b = a.clone()
    best = {t: min(_run(gb, torch, a, b, (nx, ny, nz), pitch, 0, t, 8)[1] for _ in range(8)) for t in (AUTO, SCALAR2)}
    assert best[AUTO] < 1.2 * best[SCALAR2], best  # with the asynchronous tile 1.35 to 1.58 times
