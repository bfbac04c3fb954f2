"""A domain whose time step collapses ends the run of its batch, with APPFIS_GB_ENUMERIC: after the step in
which it does, which the other domains have taken whole.  Their fields are compared bit for bit, in both state
buffers, with a run of as many steps without the collapsing domain (the two-phase pass leaves the wet/dry fix
of a run's last step to the step after it, so there the last state's momentum is not compared)."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import _lib
from appfis_gb300 import workloads as W

pytestmark = pytest.mark.gpu
ENUMERIC = 5


def _domain(gb, torch, dem, h, qx, dtype):
    real = torch.float32 if dtype == _lib.F32 else torch.float64
    ny, nx = dem.shape
    pitch = (nx + 2 + 31) // 32 * 32
    f = torch.zeros((8, ny + 2, pitch), dtype=real, device="cuda")
    d = _lib.FloodDomain()
    d.nx, d.ny, d.pitch = nx, ny, pitch
    d.h[0], d.h[1], d.qx[0], d.qx[1], d.qy[0], d.qy[1] = [f[m].data_ptr() for m in range(6)]
    d.dem, d.n2 = f[6].data_ptr(), f[7].data_ptr()
    host = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (dem, h, qx, np.zeros_like(qx))]
    gb.call("appfis_gb_flood_setup", ctypes.byref(d), dtype, *[a.data_ptr() for a in host], 0.035, None)
    torch.cuda.synchronize()
    return d, f


def _run(gb, torch, domains, dtype, flags, steps, flow=None):
    n = len(domains)
    made = [_domain(gb, torch, *d, dtype) for d in domains]
    table = (_lib.FloodDomain * n)(*[m[0] for m in made])
    prm = _lib.FloodParams(10.0, 0.5, 1e-3, 600.0, 600.0, 1.0, 0.0, steps)
    prm.flags = flags
    taken = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    status = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    out = (None, taken.data_ptr(), None, status.data_ptr(), None)
    if flow is None:
        gb.call("appfis_gb_flood_run", table, n, dtype, ctypes.byref(prm), *out)
    else:  # a point source in the last domain
        cells, times, flows = np.array([(domains[-1][0].shape[1] + 2) * 9 + 9], dtype=np.int32), np.array([0.0]), np.array([flow])
        srcs = (_lib.FloodSources * n)()
        s = srcs[n - 1]
        s.n, s.nt, s.cells, s.times, s.flows = 1, 1, cells.ctypes.data, times.ctypes.data, flows.ctypes.data
        gb.call("appfis_gb_flood_run_sources", table, srcs, n, dtype, ctypes.byref(prm), *out)
    torch.cuda.synchronize()
    return [m[1].cpu() for m in made], taken.tolist(), int(status.item())


def _healthy(side):
    dem, h = W.triton_domain(side, side + 37, side)
    h[:side // 2] += 0.5
    return dem, h, np.zeros_like(h)


def _bad(speed):
    dem, h, qx = np.zeros((20, 20)), np.full((20, 20), 0.5), np.zeros((20, 20))
    qx[3, 4] = speed
    return dem, h, qx


FORMS = [(_lib.F32, 0), (_lib.F32, _lib.FLOOD_SKIP_DRY), (_lib.F32, _lib.FLOOD_UNSTAGED), (_lib.F32, _lib.FLOOD_TWO_PHASE), (_lib.F64, 0),
         (_lib.F64, _lib.FLOOD_FUSED), (_lib.F64, _lib.FLOOD_SKIP_DRY)]


@pytest.mark.parametrize("side", [50, 700])
@pytest.mark.parametrize("dtype,flags", FORMS)
def test_the_other_domains_take_the_last_step_whole(gb, torch_cuda, dtype, flags, side):
    two_phase = flags & _lib.FLOOD_TWO_PHASE or (dtype == _lib.F64 and not flags & _lib.FLOOD_FUSED)
    want, taken, status = _run(gb, torch_cuda, [_healthy(side)], dtype, flags, 1)
    assert (taken, status) == ([1], 0)
    assert not torch_cuda.equal(want[0][0], want[0][1])
    for _ in range(3):
        got, _, status = _run(gb, torch_cuda, [_healthy(side), _bad(1e13)], dtype, flags, 5)
        assert status == ENUMERIC
        for m in ((0, 1, 2, 4) if two_phase else range(6)):  # h0 h1 qx0 qx1 qy0 qy1
            assert torch_cuda.equal(got[0][m], want[0][m]), m


@pytest.mark.parametrize("dtype,flags", [(_lib.F32, 0), (_lib.F64, 0), (_lib.F64, _lib.FLOOD_SKIP_DRY)])
def test_collapse_by_a_source_after_a_step(gb, torch_cuda, dtype, flags):
    want, taken, status = _run(gb, torch_cuda, [_healthy(700)], dtype, flags | _lib.FLOOD_TWO_PHASE, 2)
    assert (taken, status) == ([2], 0)
    for _ in range(3):
        got, taken, status = _run(gb, torch_cuda, [_healthy(700), _bad(0.0)], dtype, flags, 6, flow=1e28)
        assert status == ENUMERIC and taken == [2, 2]
        for m in (0, 1, 3, 5):  # h of both states, momentum of the first step's
            assert torch_cuda.equal(got[0][m], want[0][m]), m


@pytest.mark.parametrize("side", [50, 300])
@pytest.mark.parametrize("dtype,flags", FORMS)
def test_the_collapsing_domain_first(gb, torch_cuda, dtype, flags, side):
    """The first CTAs' strips are the collapsing domain's, so they are done at once, while others may still
    be leaving the barrier before the step."""
    two_phase = flags & _lib.FLOOD_TWO_PHASE or (dtype == _lib.F64 and not flags & _lib.FLOOD_FUSED)
    want, _, _ = _run(gb, torch_cuda, [_healthy(side)], dtype, flags, 1)
    dem, h, qx = [np.kron(a, np.ones((15, 20))) for a in _bad(1e13)]
    for _ in range(10):
        got, _, status = _run(gb, torch_cuda, [(dem, h, qx), _healthy(side)], dtype, flags, 5)
        assert status == ENUMERIC
        for m in ((0, 1, 2, 4) if two_phase else range(6)):
            assert torch_cuda.equal(got[1][m], want[0][m]), m


def test_the_next_run_is_none_the_worse(gb, torch_cuda):
    want, _, _ = _run(gb, torch_cuda, [_healthy(120)], _lib.F32, 0, 7)
    _run(gb, torch_cuda, [_healthy(120), _bad(1e13)], _lib.F32, 0, 5)
    got, taken, status = _run(gb, torch_cuda, [_healthy(120)], _lib.F32, 0, 7)
    assert (taken, status) == ([7], 0)
    for m in range(6):
        assert torch_cuda.equal(got[0][m], want[0][m]), m
