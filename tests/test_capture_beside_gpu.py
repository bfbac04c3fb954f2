"""Calls on one stream while another stream is captured into a graph, by the same thread and by another: the graph is
made and replays, and the call does what it does alone.  Every entry point that needs no workspace it does not hold."""
import ctypes
import threading

import pytest

from appfis_gb300 import _lib
from appfis_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _fields(torch, n, dtype=None, count=2):
    torch.manual_seed(7)
    return [torch.rand(n, device="cuda").to(dtype or torch.float32) for _ in range(count)]


def _life_u8(gb, torch):
    f = [(x < 0.3).to(torch.uint8) for x in _fields(torch, 2050 * 1999)]
    return f, lambda s: gb.call("appfis_gb_life_u8", f[0].data_ptr(), f[1].data_ptr(), 2050, 1999, 20, 0, None, s)


def _life_bits(gens):
    def make(gb, torch):
        f = [torch.randint(-2 ** 31, 2 ** 31 - 1, (64 * 3000,), dtype=torch.int32, device="cuda") for _ in range(2)]
        return f, lambda s: gb.call("appfis_gb_life_bits", f[0].data_ptr(), f[1].data_ptr(), 2048, 3000, gens, 0, None, s)
    return make


def _heat(gb, torch):
    f = _fields(torch, 302 * 402)
    return f, lambda s: gb.call("appfis_gb_heat2d", f[0].data_ptr(), f[1].data_ptr(), 300, 400, 302, 20, 0.2, 0.2, None, s)


def _heat64(gb, torch):
    f = _fields(torch, 302 * 402, torch.float64)
    return f, lambda s: gb.call("appfis_gb_heat2d_f64", f[0].data_ptr(), f[1].data_ptr(), 300, 400, 302, 3, 0.2, 0.2, None, s)


def _star(pitch, tile):
    def make(gb, torch):
        f, w = _fields(torch, pitch * 208 * 158), (ctypes.c_float * 5)(*W.fdtd_weights())
        return f, lambda s: gb.call("appfis_gb_star_r4", f[0].data_ptr(), f[1].data_ptr(), 0, 140, 200, 150, pitch, 2, 1, 0.1, w, tile, 0, None, s)
    return make


def _himeno(mixed, gosa):
    def make(gb, torch):
        nx, ny, nz, pitch = 40, 50, 60, 42
        f = _fields(torch, pitch * 52 * 62, count=14)
        half, g = torch.zeros(13 * f[0].numel(), dtype=torch.float16, device="cuda"), torch.zeros(6, dtype=torch.float64, device="cuda")
        c = (ctypes.c_void_p * 12)(*[x.mul_(0.1).data_ptr() for x in f[2:]])
        gp = g.data_ptr() if gosa else None
        if mixed:
            return f + [g], lambda s: gb.call("appfis_gb_himeno_mixed", c, f[0].data_ptr(), f[1].data_ptr(), half.data_ptr(), nx, ny, nz, pitch, 6, 3,
                                              0.8, gp, None, s)
        return f + [g], lambda s: gb.call("appfis_gb_himeno", c, f[0].data_ptr(), f[1].data_ptr(), nx, ny, nz, pitch, 6, 0.8, gp, None, s)
    return make


def _reduce(gb, torch):
    f, out = _fields(torch, 90 * 80 * 70, count=1), torch.zeros(1, dtype=torch.float64, device="cuda")
    box = (ctypes.c_int * 6)(1, 89, 1, 79, 1, 69)
    return f + [out], lambda s: gb.call("appfis_gb_reduce", f[0].data_ptr(), 0, 90, 80, box, 2, out.data_ptr(), s)


def _ghosts(gb, torch):
    f = _fields(torch, 90 * 80 * 70, count=1)
    return f, lambda s: gb.call("appfis_gb_ghost_periodic", f[0].data_ptr(), 4, 3, (ctypes.c_int * 3)(90, 80, 70), 2, s)


CALLS = {"life_u8": _life_u8, "life_bits 2": _life_bits(2), "life_bits 8": _life_bits(8), "life_bits 40": _life_bits(40), "heat": _heat,
         "heat_f64": _heat64, "star async": _star(150, 0), "star tma": _star(152, 0), "star scalar": _star(149, _lib.STAR_SCALAR4),
         "himeno": _himeno(False, False), "himeno gosa": _himeno(False, True), "mixed": _himeno(True, False), "reduce": _reduce, "ghosts": _ghosts}


@pytest.mark.parametrize("other_thread", [False, True])
@pytest.mark.parametrize("name", CALLS)
def test_a_capture_on_another_stream_stays_whole(gb, torch_cuda, name, other_thread):
    torch = torch_cuda
    fields, call = CALLS[name](gb, torch)
    captured, beside = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    first = [f.clone() for f in fields]
    call(beside.cuda_stream)  # alone; sizes the workspaces that some calls keep
    torch.cuda.synchronize()
    want = [f.clone() for f in fields]
    for f, v in zip(fields, first):
        f.copy_(v)
    x, graph, raised = torch.zeros(1000, device="cuda"), torch.cuda.CUDAGraph(), []

    def run():
        try:
            call(beside.cuda_stream)
        except Exception as e:  # noqa: BLE001  (reported below)
            raised.append(e)

    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=captured):
        x.add_(1)
        if other_thread:
            t = threading.Thread(target=run)
            t.start()
            t.join()
        else:
            run()
        x.add_(1)
    assert not raised, raised
    graph.replay()
    torch.cuda.synchronize()
    assert bool((x == 2).all())
    for f, v in zip(fields, want):
        assert torch.equal(f, v)
