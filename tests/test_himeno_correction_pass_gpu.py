"""The defect correction's own pass on rows that are not 16-byte aligned (a period of one sweep is nothing but such
passes): the aligned rows' fields bit for bit, heights that are no multiple of its planes per block, and its time."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _device(torch, nx, ny, nz, pitch):
    def rows(f):
        out = torch.zeros((nz + 2, ny + 2, pitch), dtype=torch.float32, device="cuda")
        out[..., :nx + 2] = torch.from_numpy(np.ascontiguousarray(f, dtype=np.float32)).cuda()
        return out
    c = [rows(f) for f in W.himeno_coef(nx, ny, nz, seed=nz)]
    p = W.himeno_p(nx, ny, nz)
    return c, (ctypes.c_void_p * 12)(*[f.data_ptr() for f in c]), rows(p), rows(p)


def _call(gb, torch, form, nx, ny, nz, pitch, iters, repeats=1):
    keep, ptrs, a, b = _device(torch, nx, ny, nz, pitch)
    half = torch.zeros(13 * a.numel(), dtype=torch.float16, device="cuda")
    gosa = torch.zeros(iters, dtype=torch.float64, device="cuda")
    ci = ctypes.c_int(-1)
    stream = torch.cuda.Stream()
    best = 1e9
    torch.cuda.synchronize()
    for _ in range(repeats):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        if form == "mixed":
            gb.call("appfis_gb_himeno_mixed", ptrs, a.data_ptr(), b.data_ptr(), half.data_ptr(), nx, ny, nz, pitch, iters, 1, 0.8,
                    gosa.data_ptr(), ctypes.byref(ci), stream.cuda_stream)
        else:
            gb.call("appfis_gb_himeno", ptrs, a.data_ptr(), b.data_ptr(), nx, ny, nz, pitch, iters, 0.8, gosa.data_ptr(), ctypes.byref(ci),
                    stream.cuda_stream)
        e1.record(stream)
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return (a if ci.value == 0 else b)[..., :nx + 2].cpu(), gosa.cpu().numpy(), best


@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (33, 5, 6), (31, 9, 7), (65, 21, 13), (20, 30, 64)])
def test_rows_of_any_alignment(gb, torch_cuda, nx, ny, nz):
    aligned = (nx + 9) // 8 * 8
    want, wg, _ = _call(gb, torch_cuda, "mixed", nx, ny, nz, aligned, 5)
    got, gg, _ = _call(gb, torch_cuda, "mixed", nx, ny, nz, aligned + 1, 5)
    assert torch_cuda.equal(got, want)
    # both sum a thread's squares in floats, at most 64 of them: 64 roundings of 2^-24
    np.testing.assert_allclose(gg, wg, rtol=64 * 2.0 ** -24)


def test_time(gb, torch_cuda):
    _, _, plain = _call(gb, torch_cuda, "plain", 65, 65, 129, 67, 20, 6)
    _, _, passes = _call(gb, torch_cuda, "mixed", 65, 65, 129, 67, 20, 6)
    assert passes < 5 * plain, (passes, plain)  # 4 times; with the coefficients asked for one by one 8 times
