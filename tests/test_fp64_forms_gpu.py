"""The FP64 sweeps' numbering of points (rows shorter than a warp, one row, planes that are no multiple
of the 4 a thread takes), their sums with and without gosa, and the doubling in the integer pipe on the
values where it has to step aside: bit for bit the oracle, or the same operations in numpy."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _heat(gb, torch, f, iters, pitch):
    host = np.full((f.shape[0], pitch), 9.0)
    host[:, : f.shape[1]] = f
    a = torch.from_numpy(host).cuda()
    b = a.clone()
    ci = ctypes.c_int(-1)
    gb.call("appfis_gb_heat2d_f64", a.data_ptr(), b.data_ptr(), f.shape[1] - 2, f.shape[0] - 2, pitch, iters, 0.2, 0.2, ctypes.byref(ci), None)
    gb.call("appfis_gb_stream_sync", None)
    return (b if ci.value else a).cpu().numpy()[:, : f.shape[1]]


@pytest.mark.parametrize("nx,ny,pitch", [(1, 1, 3), (3, 300, 8), (257, 1, 259), (31, 33, 33), (1000, 77, 1002)])
def test_heat_sizes(gb, torch_cuda, nx, ny, pitch):
    f = W.heat2d_padded(nx, ny, 1.0, nx, dtype=np.float64)
    assert np.array_equal(_heat(gb, torch_cuda, f, 5, pitch), O.heat2d(f, 5, 0.2, dtype=np.float64))


def test_heat_special_values(gb, torch_cuda):
    vals = np.array([0.0, -0.0, 5e-324, -5e-324, 2.2250738585072014e-308, 1.1e-308, -2.3e-308, 8.98846567431158e307, 8.9884656743115785e307,
                     -1.7976931348623157e308, 1.7976931348623157e308, np.inf, -np.inf, np.nan, 1.0, -3.5])
    f = vals[(W.uniform(3, 66 * 66) * len(vals)).astype(int)].reshape(66, 66)
    with np.errstate(all="ignore"):
        c = f[1:-1, 1:-1]
        two = 2.0 * c
        want = (c + 0.2 * ((f[1:-1, :-2] + f[1:-1, 2:]) - two)) + 0.2 * ((f[:-2, 1:-1] + f[2:, 1:-1]) - two)
    got = _heat(gb, torch_cuda, f, 1, 66)[1:-1, 1:-1]
    assert np.array_equal(got, want, equal_nan=True)
    assert np.array_equal(np.signbit(got[got == 0]), np.signbit(want[want == 0]))


@pytest.mark.parametrize("nx,ny,nz,pitch", [(1, 1, 1, 3), (5, 60, 3, 8), (65, 33, 10, 67), (33, 7, 41, 40)])
@pytest.mark.parametrize("with_gosa", [True, False])
def test_himeno(gb, torch_cuda, nx, ny, nz, pitch, with_gosa):
    torch, iters = torch_cuda, 3
    coef = W.himeno_coef(nx, ny, nz, dtype=np.float64, seed=nx + nz)
    p = W.himeno_p(nx, ny, nz, dtype=np.float64)
    p[1:-1, 1:-1, 1:-1] += W.uniform(3, nx * ny * nz).reshape(nz, ny, nx)

    def rows(f):
        out = torch.zeros(f.shape[:2] + (pitch,), dtype=torch.float64, device="cuda")
        out[..., : f.shape[2]] = torch.from_numpy(np.ascontiguousarray(f)).cuda()
        return out
    c = [rows(f) for f in coef]
    a, b = rows(p), rows(p)
    gosa = torch.zeros(iters, dtype=torch.float64, device="cuda")
    ci = ctypes.c_int(-1)
    gb.call("appfis_gb_himeno_f64", (ctypes.c_void_p * 12)(*[f.data_ptr() for f in c]), a.data_ptr(), b.data_ptr(), nx, ny, nz, pitch, iters, 0.8,
            gosa.data_ptr() if with_gosa else None, ctypes.byref(ci), None)
    gb.call("appfis_gb_stream_sync", None)
    ref, rg = O.himeno(coef, p, iters, 0.8, dtype=np.float64)
    assert np.array_equal((b if ci.value else a).cpu().numpy()[..., : nx + 2], ref)
    if with_gosa:
        np.testing.assert_allclose(gosa.cpu().numpy(), rg, rtol=1e-12)


@pytest.mark.parametrize("nx,ny,nz,pitch", [(1, 1, 1, 9), (3, 90, 2, 12), (33, 9, 17, 41), (70, 5, 11, 80)])
def test_star(gb, torch_cuda, nx, ny, nz, pitch):
    f = W.fdtd_padded(nx, ny, nz, nx, dtype=np.float64)
    host = np.zeros(f.shape[:2] + (pitch,))
    host[..., : nx + 8] = f
    a = torch_cuda.from_numpy(host).cuda()
    b = a.clone()
    ci = ctypes.c_int(-1)
    gb.call("appfis_gb_star_r4_f64", a.data_ptr(), b.data_ptr(), nx, ny, nz, pitch, 3, 0, 0.1, None, ctypes.byref(ci), None)
    gb.call("appfis_gb_stream_sync", None)
    got = (b if ci.value else a).cpu().numpy()[..., : nx + 8]
    g = f.copy()
    for _ in range(3):
        v = g[4:-4, 4:-4, 4:-4].copy()
        at = lambda dx, dy, dz: g[4 + dz:4 + dz + nz, 4 + dy:4 + dy + ny, 4 + dx:4 + dx + nx]  # noqa: E731
        for s in range(1, 5):
            v = v + (((at(-s, 0, 0) + at(s, 0, 0)) + (at(0, -s, 0) + at(0, s, 0))) + (at(0, 0, -s) + at(0, 0, s)))
        g[4:-4, 4:-4, 4:-4] = v * 0.1
    assert np.array_equal(got, g)
