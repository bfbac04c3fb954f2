"""Himeno routes by size and layout: the flat sweep with columns of 2, 4 and 8 planes (dense and padded rows, cut
at odd heights) and the TMA-staged sweep on a grid large enough for it, bit-identical to the oracle;
the FP16 sweep's flat form against its staged form and the FP64 oracle's bound."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _device(torch, coef, p, pitch, lead=0):
    def rows(f):
        out = torch.zeros(f.shape[0] * f.shape[1] * pitch + lead, dtype=torch.float32, device="cuda")[lead:].view(f.shape[0], f.shape[1], pitch)
        out[..., : f.shape[2]] = torch.from_numpy(np.ascontiguousarray(f, dtype=np.float32)).cuda()
        return out
    c = [rows(f) for f in coef]
    a = rows(p)
    b = rows(p)
    return c, (ctypes.c_void_p * 12)(*[f.data_ptr() for f in c]), a, b


# blocks of 256 columns: fewer than two per SM (2 planes per thread), more (4), more than ten (8), each with a
# height that is no multiple; 33 x 5 x 2 and 1 x 1 x 1; padded rows, and rows one element off 16-byte alignment;
# 190 x 190 x 170 (6.1 M points) padded is the TMA-staged form, dense the flat one
@pytest.mark.parametrize("nx,ny,nz,pitch,lead,iters", [(1, 1, 1, 3, 0, 3), (33, 5, 2, 35, 0, 4), (65, 33, 41, 67, 0, 3), (70, 70, 71, 72, 0, 3),
                                                       (70, 70, 71, 72, 1, 2), (300, 9, 130, 302, 0, 2), (151, 150, 203, 153, 0, 2),
                                                       (190, 190, 170, 192, 0, 2), (190, 190, 170, 200, 0, 3)])
@pytest.mark.parametrize("with_gosa", [True, False])
def test_plain(gb, torch_cuda, nx, ny, nz, pitch, lead, iters, with_gosa):
    torch = torch_cuda
    coef = W.himeno_coef(nx, ny, nz, seed=nx + nz)
    p = W.himeno_p(nx, ny, nz)
    p[1:-1, 1:-1, 1:-1] += W.uniform(3, nx * ny * nz).reshape(nz, ny, nx).astype(np.float32)
    keep, ptrs, a, b = _device(torch, coef, p, pitch, lead)
    gosa = torch.zeros(iters, dtype=torch.float64, device="cuda")
    ci = ctypes.c_int(-1)
    gb.call("appfis_gb_himeno", ptrs, a.data_ptr(), b.data_ptr(), nx, ny, nz, pitch, iters, 0.8, gosa.data_ptr() if with_gosa else None,
            ctypes.byref(ci), None)
    gb.call("appfis_gb_stream_sync", None)
    ref, rg = O.himeno(coef, p, iters, 0.8)
    got = (a if ci.value == 0 else b).cpu().numpy()
    assert np.array_equal(got[..., : nx + 2], ref)
    assert not got[..., nx + 2:].any()  # the padding stays as it was
    if with_gosa:
        np.testing.assert_allclose(gosa.cpu().numpy(), rg, rtol=1e-12)


@pytest.mark.parametrize("nx,ny,nz,pitch", [(65, 65, 129, 72), (33, 40, 37, 48), (100, 20, 63, 104)])
def test_mixed(gb, torch_cuda, nx, ny, nz, pitch):
    """Without gosa a small grid takes the flat sweep: the same p bit for bit as the staged sweep with
    gosa.  Dense rows (flat in either case) stay within the mixed form's 2.5e-4 of the FP64 oracle."""
    torch = torch_cuda
    iters, period = 25, 10
    coef, p = W.himeno_coef(nx, ny, nz), W.himeno_p(nx, ny, nz)
    out = {}
    for key, pt, with_gosa in (("staged", pitch, True), ("flat", pitch, False), ("dense", nx + 2, True)):
        keep, ptrs, a, b = _device(torch, coef, p, pt)
        half = torch.empty(13 * a.numel(), dtype=torch.float16, device="cuda")
        gosa = torch.zeros(iters, dtype=torch.float64, device="cuda")
        ci = ctypes.c_int(-1)
        gb.call("appfis_gb_himeno_mixed", ptrs, a.data_ptr(), b.data_ptr(), half.data_ptr(), nx, ny, nz, pt, iters, period, 0.8,
                gosa.data_ptr() if with_gosa else None, ctypes.byref(ci), None)
        gb.call("appfis_gb_stream_sync", None)
        out[key] = ((a if ci.value == 0 else b).cpu().numpy()[..., : nx + 2], gosa.cpu().numpy())
    assert np.array_equal(out["flat"][0], out["staged"][0])
    p64, g64 = O.himeno(W.himeno_coef(nx, ny, nz, dtype=np.float64), W.himeno_p(nx, ny, nz, dtype=np.float64), iters, 0.8, dtype=np.float64)
    assert np.abs(out["dense"][0] - p64).max() < 2.5e-4
    np.testing.assert_allclose(out["dense"][1], g64, rtol=1e-2)
