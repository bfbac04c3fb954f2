"""A flood run's tables (domains, row maps, point sources) are the library's from the moment the call returns:
runs queued one after the other behind a busy stream, whose host tables are long gone and overwritten when the
stream reaches them, give what each gives alone.  More of them than the library stages at once, and one whose
source table is larger than a staging buffer."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import _lib
from appfis_gb300 import workloads as W

pytestmark = pytest.mark.gpu
STEPS = 6


class _Run:
    def __init__(self, gb, torch, domains, dtype, rows):
        real = torch.float32 if dtype == _lib.F32 else torch.float64
        n = len(domains)
        self.n, self.dtype, self.rows = n, dtype, rows
        self.shapes, self.fields = [d[0].shape for d in domains], []
        self.status = torch.full((1,), -1, dtype=torch.int32, device="cuda")
        table = self.table()
        for k, (dem, h) in enumerate(domains):
            f = torch.zeros((8, dem.shape[0] + 2, table[k].pitch), dtype=real, device="cuda")
            self.fields.append(f)
            d = self.table()[k]
            dd, hh = torch.from_numpy(dem).cuda(), torch.from_numpy(h).cuda()
            gb.call("appfis_gb_flood_setup", ctypes.byref(d), dtype, dd.data_ptr(), hh.data_ptr(), None, None, 0.035, None)
            torch.cuda.synchronize()

    def table(self):
        t = (_lib.FloodDomain * self.n)()
        for k, (ny, nx) in enumerate(self.shapes):
            d = t[k]
            d.nx, d.ny, d.pitch = nx, ny, (nx + 2 + 31) // 32 * 32
            if k < len(self.fields):
                f = self.fields[k]
                d.h[0], d.h[1], d.qx[0], d.qx[1], d.qy[0], d.qy[1] = [f[m].data_ptr() for m in range(6)]
                d.dem, d.n2 = f[6].data_ptr(), f[7].data_ptr()
        return t

    def go(self, gb, stream):
        """The caller's tables are wiped as soon as the call returns."""
        t, prm = self.table(), _lib.FloodParams(10.0, 0.5, 1e-3, 600.0, 600.0, 1.0, 0.0, STEPS)
        if self.rows:
            cells = np.array([2 * (self.shapes[0][1] + 2) + 3], dtype=np.int32)
            times, flows = np.arange(self.rows, dtype=np.float64), np.linspace(50.0, 90.0, self.rows)
            s = (_lib.FloodSources * self.n)()
            s[0].n, s[0].nt, s[0].cells, s[0].times, s[0].flows = 1, self.rows, cells.ctypes.data, times.ctypes.data, flows.ctypes.data
            gb.call("appfis_gb_flood_run_sources", t, s, self.n, self.dtype, ctypes.byref(prm), None, None, None, self.status.data_ptr(), stream)
            cells[:], times[:], flows[:] = -1, -1.0, -1.0
        else:
            gb.call("appfis_gb_flood_run", t, self.n, self.dtype, ctypes.byref(prm), None, None, None, self.status.data_ptr(), stream)
        ctypes.memset(t, 0, ctypes.sizeof(t))


def _runs(gb, torch):
    out = []
    for k in range(7):
        shapes = [(30 + 7 * k, 41 + 11 * k)] + [(20 + k, 33 + j) for j in range(k)]
        doms = [W.triton_domain(ny, nx, 100 * k + i) for i, (ny, nx) in enumerate(shapes)]
        out.append(_Run(gb, torch, doms, _lib.F64 if k % 3 == 2 else _lib.F32, (0, 0, 3, 0, 20000, 0, 5)[k]))
    return out


def test_runs_queued_behind_a_busy_stream(gb, torch_cuda):
    torch = torch_cuda
    alone = _runs(gb, torch)
    for r in alone:
        r.go(gb, None)
        torch.cuda.synchronize()
    queued = _runs(gb, torch)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(50000000)  # some 25 ms
        for r in queued:
            r.go(gb, stream.cuda_stream)
    torch.cuda.synchronize()
    for a, q in zip(alone, queued):
        assert int(a.status.item()) == int(q.status.item()) == 0
        for x, y in zip(a.fields, q.fields):
            assert torch.equal(x, y)
            assert not torch.equal(x[0], x[1])


def test_the_host_goes_on(gb, torch_cuda):
    """One run does not wait for what is before it on its stream."""
    torch = torch_cuda
    r = _runs(gb, torch)[1]
    r.go(gb, None)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    done = torch.cuda.Event()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(200000000)  # some 100 ms
        done.record()
        r.go(gb, stream.cuda_stream)
        assert not done.query()
    torch.cuda.synchronize()
    assert int(r.status.item()) == 0
