"""The size rules of the GameOfLife runs against the oracle: tile heights of the time-blocked kernel, the
split of a run into launches, byte rows of any length and alignment through the packed form, and
the sweeps that the shortest runs take.  States are whole numbers: every cell equal."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _oracle(cells, gens, rule):
    """(state, state before it or None where the oracle does not give it)"""
    return O.gol(cells, gens) if rule == 0 else (O.gol_b3s23(cells, gens), O.gol_b3s23(cells, gens - 1))


# tiles of 32 rows (small), 64 and 128 rows (19200 cells = 20 tile columns; 760 and 1530 rows), each
# with a last tile that is cut; 1 to 3 generations as sweeps, 4 to 15 in two launches, 16 to 33 in two or three
@pytest.mark.parametrize("nx,ny,gens", [(32, 3, 4), (64, 31, 5), (992, 33, 15), (1024, 65, 16), (1024, 100, 17), (96, 200, 33), (2048, 50, 3),
                                        (19200, 760, 5), (19200, 1530, 4)])
@pytest.mark.parametrize("rule", [0, 1])
def test_bits(gb, torch_cuda, nx, ny, gens, rule):
    cells = W.gol_cells(nx, ny, 0.3, nx + ny)
    c = torch_cuda.from_numpy(cells).cuda()
    a = torch_cuda.empty(ny, nx // 32, dtype=torch_cuda.int32, device="cuda")
    buf = [a, torch_cuda.zeros_like(a)]
    gb.call("appfis_gb_life_pack", c.data_ptr(), a.data_ptr(), nx, ny, None)
    ci = ctypes.c_int(-1)
    gb.call("appfis_gb_life_bits", buf[0].data_ptr(), buf[1].data_ptr(), nx, ny, gens, rule, ctypes.byref(ci), None)
    assert ci.value == gens % 2
    for got, want in zip((buf[ci.value], buf[1 - ci.value]), _oracle(cells, gens, rule)):
        gb.call("appfis_gb_life_unpack", got.data_ptr(), c.data_ptr(), nx, ny, None)
        gb.call("appfis_gb_stream_sync", None)
        assert np.array_equal(c.cpu().numpy(), want)


# rows one short of, at and past whole words and tile columns (960 cells), the smallest width, buffers
# at every alignment; a grid of 4 M cells at 1 to 3 generations (one thread per cell, bulk, packed)
@pytest.mark.parametrize("nx,ny,gens,lead", [(64, 9, 9, 0), (65, 70, 17, 1), (63, 20, 6, 0), (95, 33, 4, 2), (97, 1, 33, 3), (959, 40, 16, 5),
                                             (961, 41, 5, 0), (1001, 300, 16, 9), (1936, 64, 12, 0), (2050, 97, 40, 0), (2080, 64, 7, 0),
                                             (4112, 1030, 1, 0), (4112, 1030, 3, 0), (4100, 1030, 1, 0), (4100, 1030, 2, 7)])
@pytest.mark.parametrize("rule", [0, 1])
def test_u8(gb, torch_cuda, nx, ny, gens, lead, rule):
    cells = W.gol_cells(nx, ny, 0.35, nx + ny)
    n = nx * ny
    guard = torch_cuda.full((2, lead + n + 32), 7, dtype=torch_cuda.uint8, device="cuda")  # bytes around each plane stay
    planes = [guard[k, lead:lead + n] for k in range(2)]
    store = [p.clone() for p in planes] if nx % 16 == 0 else planes  # whole 16-byte rows come in aligned buffers
    store[0].copy_(torch_cuda.from_numpy(cells).reshape(-1).cuda())
    store[1].zero_()
    ci = ctypes.c_int(-1)
    gb.call("appfis_gb_life_u8", store[0].data_ptr(), store[1].data_ptr(), nx, ny, gens, rule, ctypes.byref(ci), None)
    gb.call("appfis_gb_stream_sync", None)
    assert ci.value == gens % 2
    for got, want in zip((store[ci.value], store[1 - ci.value]), _oracle(cells, gens, rule)):
        assert np.array_equal(got.cpu().numpy().reshape(ny, nx), want)
    assert bool((guard[:, :lead] == 7).all()) and bool((guard[:, lead + n:] == 7).all())


def test_u8_while_recording_a_graph(gb, torch_cuda):
    """A recorded run takes the sweeps, which need no memory of their own, and replays to the same state."""
    nx, ny, gens = 301, 70, 12
    cells = W.gol_cells(nx, ny, 0.3, 5)
    a = torch_cuda.from_numpy(cells).cuda()
    b = torch_cuda.zeros_like(a)
    ci, g = ctypes.c_int(-1), torch_cuda.cuda.CUDAGraph()
    with torch_cuda.cuda.graph(g):
        gb.call("appfis_gb_life_u8", a.data_ptr(), b.data_ptr(), nx, ny, gens, 0, ctypes.byref(ci),
                torch_cuda.cuda.current_stream().cuda_stream)
    g.replay()
    torch_cuda.cuda.synchronize()
    assert np.array_equal((b if ci.value else a).cpu().numpy(), O.gol(cells, gens)[0])
