"""FP64 Himeno with 1 to 4 planes per thread, by size and with and without gosa: the oracle's fields bit for bit, and
a small grid in the time of its blocks beside one another."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _run(gb, torch, nx, ny, nz, iters, with_gosa, repeats=1):
    coef, p = W.himeno_coef(nx, ny, nz, seed=3, dtype=np.float64), W.himeno_p(nx, ny, nz, dtype=np.float64)
    c = [torch.from_numpy(np.ascontiguousarray(f)).cuda() for f in coef]
    a = torch.from_numpy(np.ascontiguousarray(p)).cuda()
    b = a.clone()
    gosa = torch.zeros(iters, dtype=torch.float64, device="cuda")
    ptrs, ci, stream, best = (ctypes.c_void_p * 12)(*[f.data_ptr() for f in c]), ctypes.c_int(-1), torch.cuda.Stream(), 1e9
    torch.cuda.synchronize()
    for _ in range(repeats):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        gb.call("appfis_gb_himeno_f64", ptrs, a.data_ptr(), b.data_ptr(), nx, ny, nz, nx + 2, iters, 0.8, gosa.data_ptr() if with_gosa else None,
                ctypes.byref(ci), stream.cuda_stream)
        e1.record(stream)
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return coef, p, (a if ci.value == 0 else b).cpu().numpy(), gosa.cpu().numpy(), best


# on 152 SMs with gosa 1, 3, 2, 4 and 4 planes per thread, heights that are no multiple
@pytest.mark.parametrize("nx,ny,nz", [(24, 24, 23), (33, 33, 65), (64, 64, 127), (65, 65, 63), (129, 129, 30), (1, 1, 5)])
@pytest.mark.parametrize("with_gosa", [True, False])
def test_fields_and_gosa(gb, torch_cuda, nx, ny, nz, with_gosa):
    coef, p, got, gosa, _ = _run(gb, torch_cuda, nx, ny, nz, 3, with_gosa)
    want, wg = O.himeno(coef, p, 3, 0.8, dtype=np.float64)
    assert np.array_equal(got, want)
    if with_gosa:
        np.testing.assert_allclose(gosa, wg, rtol=1e-12)


def test_a_small_grid_is_spread_out(gb, torch_cuda):
    *_, t = _run(gb, torch_cuda, 24, 24, 24, 50, False, 6)
    *_, one = _run(gb, torch_cuda, 24, 24, 1, 50, False, 6)
    assert t < 2 * one, (t, one)  # 72 blocks of a plane on 152 SMs take as long as 3 do; with 4 planes per thread 2.9 times
