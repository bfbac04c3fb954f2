"""The TMA-staged Himeno sweep (16-byte rows, more than 6 M points) on ragged x tiles, cut y tiles and short z chunks:
the dense rows' fields (the flat sweep) bit for bit, gosa to 1e-12, padding as it was."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _run(gb, torch, coef, p, nx, ny, nz, pitch, iters):
    def rows(f):
        out = torch.full((nz + 2, ny + 2, pitch), 3.0, dtype=torch.float32, device="cuda")
        out[..., :nx + 2] = f
        return out
    c = [rows(f) for f in coef]
    a, b = rows(p), rows(p)
    gosa, ci = torch.zeros(iters, dtype=torch.float64, device="cuda"), ctypes.c_int(-1)
    torch.cuda.synchronize()
    gb.call("appfis_gb_himeno", (ctypes.c_void_p * 12)(*[f.data_ptr() for f in c]), a.data_ptr(), b.data_ptr(), nx, ny, nz, pitch, iters, 0.8,
            gosa.data_ptr(), ctypes.byref(ci), None)
    gb.call("appfis_gb_stream_sync", None)
    got = a if ci.value == 0 else b
    assert bool((got[..., nx + 2:] == 3.0).all())
    return got[..., :nx + 2], gosa.cpu().numpy()


@pytest.mark.parametrize("nx,ny,nz,pitch", [(30, 451, 450, 32), (31, 500, 400, 36), (33, 500, 389, 36), (64, 331, 300, 68), (65, 310, 310, 68),
                                            (255, 201, 130, 260), (1000, 789, 8, 1004), (257, 25, 1000, 260), (600, 7, 1500, 604), (1, 3000, 2100, 4),
                                            (2000, 3001, 1, 2004), (95, 260, 250, 100)])
def test_ragged_tiles(gb, torch_cuda, nx, ny, nz, pitch):
    torch = torch_cuda
    assert nx * ny * nz > 6000000 and pitch % 4 == 0
    torch.manual_seed(nx)
    coef = [torch.rand((nz + 2, ny + 2, nx + 2), device="cuda") * 0.1 + 0.1 for _ in range(12)]
    p = torch.rand((nz + 2, ny + 2, nx + 2), device="cuda")
    got, gg = _run(gb, torch, coef, p, nx, ny, nz, pitch, 3)
    dense = nx + 2 if (nx + 2) % 4 else nx + 3  # rows that are not 16-byte aligned
    want, wg = _run(gb, torch, coef, p, nx, ny, nz, dense, 3)
    assert torch.equal(got, want)
    np.testing.assert_allclose(gg, wg, rtol=1e-12)
