"""The order in which a flood step takes its strips: a batch of fewer than two strips per resident warp takes
them as numbered, a larger one the wet strips of the step before first, the dry ones behind.  With a
point source that wets dry ground, both passes, FP32 and FP64 and dry strips left out or not, a domain's
fields, steps and time steps are the same alone and beside a large domain; bit for bit, as the order only
shares out strips that do not depend on each other."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import _lib
from appfis_gb300 import workloads as W

pytestmark = pytest.mark.gpu
STEPS = 26


def _run(gb, torch, domains, dtype, flags, source):
    real = torch.float32 if dtype == _lib.F32 else torch.float64
    n = len(domains)
    table, srcs, keep = (_lib.FloodDomain * n)(), (_lib.FloodSources * n)(), []
    for k, (dem, h) in enumerate(domains):
        ny, nx = dem.shape
        pitch = (nx + 2 + 31) // 32 * 32
        f = torch.zeros((8, ny + 2, pitch), dtype=real, device="cuda")
        d = table[k]
        d.nx, d.ny, d.pitch = nx, ny, pitch
        d.h[0], d.h[1], d.qx[0], d.qx[1], d.qy[0], d.qy[1] = [f[m].data_ptr() for m in range(6)]
        d.dem, d.n2 = f[6].data_ptr(), f[7].data_ptr()
        dd, hh = torch.from_numpy(dem).cuda(), torch.from_numpy(h).cuda()
        gb.call("appfis_gb_flood_setup", ctypes.byref(d), dtype, dd.data_ptr(), hh.data_ptr(), None, None, 0.035, None)
        torch.cuda.synchronize()
        if source:
            cells = np.array([(ny // 3 + 1) * (nx + 2) + nx // 2, (ny - 1) * (nx + 2) + 2], dtype=np.int32)
            times, flows = np.array([0.0, 1e4]), np.array([[20.0, 5.0], [60.0, 9.0]])
            s = srcs[k]
            s.n, s.nt, s.cells, s.times, s.flows = 2, 2, cells.ctypes.data, times.ctypes.data, flows.ctypes.data
            keep.append((cells, times, flows))
        keep.append(f)
    prm = _lib.FloodParams(10.0, 0.5, 1e-3, 600.0, 600.0, 1.0, 0.0, STEPS)
    prm.flags = flags
    steps = torch.zeros(n, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    dts = torch.zeros(n * STEPS, dtype=torch.float64, device="cuda")
    if source:
        gb.call("appfis_gb_flood_run_sources", table, srcs, n, dtype, ctypes.byref(prm), dts.data_ptr(), steps.data_ptr(), None,
                status.data_ptr(), None)
    else:
        gb.call("appfis_gb_flood_run", table, n, dtype, ctypes.byref(prm), dts.data_ptr(), steps.data_ptr(), None, status.data_ptr(), None)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    fields = [a for a in keep if isinstance(a, torch.Tensor)]
    out = []
    for k, (dem, _) in enumerate(domains):
        b = int(steps[k].item()) & 1
        out.append([fields[k][2 * m + b][1:dem.shape[0] + 1, 1:dem.shape[1] + 1].cpu() for m in range(3)])
    return out, steps.cpu()


@pytest.mark.parametrize("source", [False, True])
@pytest.mark.parametrize("flags", [0, _lib.FLOOD_SKIP_DRY, _lib.FLOOD_TWO_PHASE, _lib.FLOOD_TWO_PHASE | _lib.FLOOD_SKIP_DRY])
@pytest.mark.parametrize("dtype,beside", [(_lib.F32, 1100), (_lib.F32, 3300), (_lib.F64, 640), (_lib.F64, 1500)])
def test_fields_do_not_depend_on_the_order(gb, torch_cuda, dtype, beside, flags, source):
    small = [W.triton_domain(ny, nx, 900 + nx) for ny, nx in ((41, 127), (2, 3), (95, 61))]
    rng = np.random.default_rng(beside)
    dem, h = rng.random((beside, beside)), np.zeros((beside, beside))
    for y, x in rng.integers(0, beside - 40, (12, 2)):  # wet spots among dry strips
        h[y:y + 30, x:x + 40] = 0.7
    alone, sa = _run(gb, torch_cuda, small, dtype, flags, source)
    batch, sb = _run(gb, torch_cuda, small + [(dem, h)], dtype, flags, source)
    assert torch_cuda.equal(sa, sb[:len(small)])
    for k in range(len(small)):
        for a, b in zip(alone[k], batch[k]):
            assert torch_cuda.equal(a, b), k
    assert all(f[0].abs().sum() > 0 for f in batch)


def test_capturing_stream_is_refused(gb, torch_cuda):
    """A run copies tables from the caller's memory, which a graph could not replay: an error, and the
    stream and the next run are none the worse."""
    torch = torch_cuda
    domains = [W.triton_domain(20, 30, 5)]
    want, _ = _run(gb, torch, domains, _lib.F32, 0, False)
    table, prm = (_lib.FloodDomain * 1)(), _lib.FloodParams(10.0, 0.5, 1e-3, 600.0, 600.0, 1.0, 0.0, STEPS)
    f = torch.zeros((8, 22, 32), device="cuda")
    table[0].nx, table[0].ny, table[0].pitch = 30, 20, 32
    table[0].h[0], table[0].h[1], table[0].qx[0], table[0].qx[1], table[0].qy[0], table[0].qy[1] = [f[m].data_ptr() for m in range(6)]
    table[0].dem, table[0].n2 = f[6].data_ptr(), f[7].data_ptr()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        with pytest.raises(_lib.AppfisError):
            gb.call("appfis_gb_flood_run", table, 1, _lib.F32, ctypes.byref(prm), None, None, None, None, torch.cuda.current_stream().cuda_stream)
    got, _ = _run(gb, torch, domains, _lib.F32, 0, False)
    for a, b in zip(got[0], want[0]):
        assert torch.equal(a, b)
