"""Every band height of the time-blocked GameOfLife kernel, with the words left over in columns of their own and side by
side, whole and ragged words, both rules: against the one-generation kernels (bit-packed sweeps; byte sweeps,
which a recorded run takes), every cell of both states equal.  The sizes are the smallest of a few families for
which the size rule of the device at hand takes each height; and the two large grids of the workloads."""
import ctypes
import functools

import pytest

pytestmark = pytest.mark.gpu
BANDS = (5, 6, 7, 8, 10, 12, 14, 16, 18, 20, 22, 24, 26, 28, 30, 33, 36, 39, 41, 43, 45)


def _plan(nw, ny, sms):
    """The library's choice for rows of nw words: (rows per band, words left over side by side)."""
    best, cost = None, 1e30
    for beside in range(2 if nw % 30 and nw % 30 <= 14 else 1):
        for band in BANDS:
            high = -(-ny // (8 * band - 32))
            cols, rest = (nw // 30, nw % 30) if beside else (-(-nw // 30), 0)
            tiles = cols * high + (-(-high // (32 // (rest + 2))) if rest else 0)
            c = -(-tiles // sms) * (0.47 * band + 0.2)
            if beside:
                c = max(1.05 * c, c + 0.8)
            if c < cost or (c == cost and not beside):
                best, cost = (band, bool(beside)), c
    return best


@functools.lru_cache(None)
def _sizes(sms):
    found = {}
    for nw in (17, 30, 31, 33, 35, 45, 60, 61, 64, 70, 90, 100, 150, 240, 310, 360, 480, 500, 510, 512):
        for k in range(170):
            ny = int(100 * 1.035 ** k) + k % 3
            if nw * ny * 32 > 3e8:
                break
            p = _plan(nw, ny, sms)
            if p not in found or nw * ny < found[p][0] * found[p][1]:
                found[p] = (nw, ny)
    return found


def _bits_call(gb, a, b, nx, ny, gens, rule):
    ci = ctypes.c_int(-1)
    gb.call("appfis_gb_life_bits", a.data_ptr(), b.data_ptr(), nx, ny, gens, rule, ctypes.byref(ci), None)
    return (a, b) if ci.value == 0 else (b, a)


def _check_bits(gb, torch, nw, ny, rule, runs):
    a = torch.randint(-2 ** 31, 2 ** 31 - 1, (ny * nw,), dtype=torch.int32, device="cuda") & torch.randint(-2 ** 31, 2 ** 31 - 1, (ny * nw,), dtype=torch.int32, device="cuda")
    b = torch.randint(-2 ** 31, 2 ** 31 - 1, (ny * nw,), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    got, want = (a.clone(), b.clone()), (a, b)
    for gens in runs:
        got = _bits_call(gb, *got, 32 * nw, ny, gens, rule)
        for _ in range(gens):
            want = _bits_call(gb, *want, 32 * nw, ny, 1, rule)
        gb.call("appfis_gb_stream_sync", None)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), gens


@pytest.mark.parametrize("rule", [0, 1])
@pytest.mark.parametrize("beside", [False, True])
@pytest.mark.parametrize("band", BANDS)
def test_every_band(gb, torch_cuda, band, beside, rule):
    torch = torch_cuda
    size = _sizes(torch.cuda.get_device_properties(0).multi_processor_count).get((band, beside))
    if size is None:
        pytest.skip("no size takes it on this device")
    nw, ny = size
    torch.manual_seed(band)
    _check_bits(gb, torch, nw, ny, rule, (32, 7))  # launches of 16 generations, of 3 and 4
    # ragged rows of as many words: the packed byte run against the byte sweeps of a recorded one
    nx = 32 * nw - 13
    cells = [(torch.rand(ny * nx, device="cuda") < 0.3).to(torch.uint8) for _ in range(2)]
    copies = [c.clone() for c in cells]
    ci, graph = ctypes.c_int(-1), torch.cuda.CUDAGraph()
    gb.call("appfis_gb_life_u8", cells[0].data_ptr(), cells[1].data_ptr(), nx, ny, 19, rule, ctypes.byref(ci), None)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        gb.call("appfis_gb_life_u8", copies[0].data_ptr(), copies[1].data_ptr(), nx, ny, 19, rule, ctypes.byref(ci),
                torch.cuda.current_stream().cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(cells[0], copies[0]) and torch.equal(cells[1], copies[1])


@pytest.mark.parametrize("rule", [0, 1])
@pytest.mark.parametrize("nw,ny", [(497, 12000), (512, 16384), (128, 4096), (256, 8192)])
def test_large_grids(gb, torch_cuda, nw, ny, rule):
    torch_cuda.manual_seed(ny)
    _check_bits(gb, torch_cuda, nw, ny, rule, (45, 4))
