"""Rows far longer in memory than the grid is wide (a grid inside a larger allocation): the flat sweeps, plain and
FP16, and the last pass of the defect correction give the dense rows' results bit for bit, touch
no padding, and take no time for it."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _fields(torch, nx, ny, nz, pitch):
    def rows(f):
        out = torch.full((nz + 2, ny + 2, pitch), 7.0, dtype=torch.float32, device="cuda")
        out[..., :nx + 2] = torch.from_numpy(np.ascontiguousarray(f, dtype=np.float32)).cuda()
        return out
    c = [rows(f) for f in W.himeno_coef(nx, ny, nz, seed=5)]
    p = W.himeno_p(nx, ny, nz)
    return c, (ctypes.c_void_p * 12)(*[f.data_ptr() for f in c]), rows(p), rows(p)


def _plain(gb, torch, nx, ny, nz, pitch, iters, time=False):
    keep, ptrs, a, b = _fields(torch, nx, ny, nz, pitch)
    gosa = torch.zeros(iters, dtype=torch.float64, device="cuda")
    ci = ctypes.c_int(-1)
    args = (ptrs, a.data_ptr(), b.data_ptr(), nx, ny, nz, pitch, iters, 0.8, gosa.data_ptr(), ctypes.byref(ci))
    stream = torch.cuda.Stream()
    best = None
    torch.cuda.synchronize()
    for _ in range(6 if time else 1):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        gb.call("appfis_gb_himeno", *args, stream.cuda_stream)
        e1.record(stream)
        torch.cuda.synchronize()
        best = min(best or 1e9, e0.elapsed_time(e1))
    return (a if ci.value == 0 else b).cpu(), gosa.cpu(), best


@pytest.mark.parametrize("nx,ny,nz,pitch", [(1, 1, 1, 300), (30, 21, 40, 1024), (65, 33, 41, 1001), (2, 80, 90, 513)])
def test_plain(gb, torch_cuda, nx, ny, nz, pitch):
    want, wg, _ = _plain(gb, torch_cuda, nx, ny, nz, nx + 2, 3)
    got, gg, _ = _plain(gb, torch_cuda, nx, ny, nz, pitch, 3)
    assert torch_cuda.equal(got[..., :nx + 2], want)
    assert torch_cuda.all(got[..., nx + 2:] == 7.0)
    assert torch_cuda.equal(gg, wg)  # the points are numbered alike, so the squares are summed alike


@pytest.mark.parametrize("nx,ny,nz,pitch", [(1, 1, 1, 301), (30, 21, 40, 1023), (65, 33, 41, 1001)])
def test_mixed(gb, torch_cuda, nx, ny, nz, pitch):
    torch = torch_cuda
    out = []
    for pt in (nx + 2 + (nx & 1), pitch):  # the flat form but for 32, where it is the staged one, which sums its squares in floats
        keep, ptrs, a, b = _fields(torch, nx, ny, nz, pt)
        half = torch.zeros(13 * a.numel(), dtype=torch.float16, device="cuda")
        gosa = torch.zeros(7, dtype=torch.float64, device="cuda")
        ci = ctypes.c_int(-1)
        gb.call("appfis_gb_himeno_mixed", ptrs, a.data_ptr(), b.data_ptr(), half.data_ptr(), nx, ny, nz, pt, 7, 3, 0.8, gosa.data_ptr(),
                ctypes.byref(ci), None)
        gb.call("appfis_gb_stream_sync", None)
        out.append(((a if ci.value == 0 else b)[:, 1:ny + 1, 1:nx + 1].cpu(), gosa.cpu()))
    assert torch.equal(out[0][0], out[1][0])
    if nx != 30:
        assert torch.equal(out[0][1], out[1][1])


def test_padding_takes_no_time(gb, torch_cuda):
    _, _, dense = _plain(gb, torch_cuda, 30, 200, 200, 32, 20, time=True)
    _, _, wide = _plain(gb, torch_cuda, 30, 200, 200, 4096, 20, time=True)
    assert wide < 5 * dense, (wide, dense)  # 1.4 times (its lines hold a quarter as much); with the padding numbered 16 times
