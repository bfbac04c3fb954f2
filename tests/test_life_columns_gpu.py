"""Grids whose rows leave a few words over from whole tile columns, tall enough that the time-blocked kernel sets
several tiles of those words side by side in a warp: 1 to 13 words left, beside whole columns or alone,
whole and ragged words, rows that end inside a tile, against the oracle; every cell equal."""
import ctypes

import numpy as np
import pytest

from appfis_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# words a row: 31 (one left, ten tiles beside one another), 3 (alone), 43 (13 left, two tiles), 31, 3, 65, 14
@pytest.mark.parametrize("nx,ny,gens", [(992, 5000, 17), (96, 33000, 5), (1376, 5003, 16), (970, 5001, 33), (70, 20011, 6), (2050, 3999, 16),
                                        (447, 9001, 4)])
@pytest.mark.parametrize("rule", [0, 1])
def test_words_left_over(gb, torch_cuda, nx, ny, gens, rule):
    cells = W.gol_cells(nx, ny, 0.33, nx + ny)
    a = torch_cuda.from_numpy(cells).cuda()
    buf = [a, torch_cuda.zeros_like(a)]
    ci = ctypes.c_int(-1)
    gb.call("appfis_gb_life_u8", buf[0].data_ptr(), buf[1].data_ptr(), nx, ny, gens, rule, ctypes.byref(ci), None)
    gb.call("appfis_gb_stream_sync", None)
    want = O.gol(cells, gens) if rule == 0 else (O.gol_b3s23(cells, gens), O.gol_b3s23(cells, gens - 1))
    for got, state in zip((buf[ci.value], buf[1 - ci.value]), want):
        assert np.array_equal(got.cpu().numpy(), state)
