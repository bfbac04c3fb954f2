"""The byte-per-cell GameOfLife sweep whose rows are staged by bulk copies: what a recorded run of 4 M cells in rows of
whole 16-byte vectors takes, and a single generation of 8 M.  Strips of 4096 cells alone, cut and with a
short one beside them, heights that are no multiple of 32, against the oracle; every cell of both states equal."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _want(cells, gens, rule):
    return O.gol(cells, gens) if rule == 0 else (O.gol_b3s23(cells, gens), O.gol_b3s23(cells, gens - 1))


@pytest.mark.parametrize("nx,ny,gens", [(4096, 1024, 5), (4112, 1030, 3), (16, 262147, 3), (48, 87391, 4), (8704, 483, 6), (2048, 2049, 7),
                                        (4080, 1033, 2)])
@pytest.mark.parametrize("rule", [0, 1])
def test_recorded(gb, torch_cuda, nx, ny, gens, rule):
    torch = torch_cuda
    cells = W.gol_cells(nx, ny, 0.3, nx)
    a = torch.from_numpy(cells).cuda()
    b = torch.zeros_like(a)
    ci, graph = ctypes.c_int(-1), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    # the status word of the staged sweeps exists from the first of them on
    warm = [torch.zeros(4096 * 2048, dtype=torch.uint8, device="cuda") for _ in range(2)]
    gb.call("appfis_gb_life_u8", warm[0].data_ptr(), warm[1].data_ptr(), 4096, 2048, 1, rule, ctypes.byref(ci), None)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        gb.call("appfis_gb_life_u8", a.data_ptr(), b.data_ptr(), nx, ny, gens, rule, ctypes.byref(ci), torch.cuda.current_stream().cuda_stream)
    assert ci.value == gens % 2
    graph.replay()
    gb.call("appfis_gb_stream_sync", None)
    torch.cuda.synchronize()
    for got, want in zip((a, b) if ci.value == 0 else (b, a), _want(cells, gens, rule)):
        assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("nx,ny", [(4096, 2048), (4112, 2051), (64, 131100), (12304, 700)])
@pytest.mark.parametrize("rule", [0, 1])
def test_one_generation(gb, torch_cuda, nx, ny, rule):
    torch = torch_cuda
    cells, old = W.gol_cells(nx, ny, 0.35, ny), W.gol_cells(nx, ny, 0.5, 3)
    a, b = torch.from_numpy(cells).cuda(), torch.from_numpy(old).cuda()
    ci = ctypes.c_int(-1)
    gb.call("appfis_gb_life_u8", a.data_ptr(), b.data_ptr(), nx, ny, 1, rule, ctypes.byref(ci), None)
    gb.call("appfis_gb_stream_sync", None)
    assert ci.value == 1
    want = O.gol(cells, 1, old=old)[0] if rule == 0 else O.gol_b3s23(cells, 1)
    assert np.array_equal(b.cpu().numpy(), want)
    assert np.array_equal(a.cpu().numpy(), cells)
