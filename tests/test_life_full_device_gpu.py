"""Bit-packed runs whose launches would be odd in number (33 to 47 generations, 65 to 79 ...) use a third pair of planes;
on a device that has no room for it they run without, with the same states, and give back the plane they had.
In a process of its own, as the library keeps the planes of earlier, smaller runs."""
import ctypes
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
NX, NY = 65536, 32768
PLANE = NX * NY // 8


def _state(torch, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    a = torch.randint(-2 ** 31, 2 ** 31 - 1, (PLANE // 4,), dtype=torch.int32, device="cuda", generator=g)
    b = torch.zeros_like(a)
    torch.cuda.synchronize()
    return a, b


def _child(gens):
    import torch

    import appfis_gb300 as gb
    ci = ctypes.c_int(-1)
    states = [_state(torch, 5) for _ in range(2)]
    a, b = states[0]
    for n in (16, gens - 16):  # an even number of launches each: the two pairs, now sized
        gb.call("appfis_gb_life_bits", a.data_ptr(), b.data_ptr(), NX, NY, n, 0, ctypes.byref(ci), None)
        assert ci.value == 0
    gb.call("appfis_gb_stream_sync", None)
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - PLANE - PLANE // 2, dtype=torch.uint8, device="cuda")  # room for one plane more, not for two
    c, d = states[1]
    gb.call("appfis_gb_life_bits", c.data_ptr(), d.data_ptr(), NX, NY, gens, 0, ctypes.byref(ci), None)
    gb.call("appfis_gb_stream_sync", None)
    assert torch.cuda.mem_get_info()[0] >= PLANE  # the first plane of the pair was given back
    del hold
    assert ci.value == 0
    assert torch.equal(a, c) and torch.equal(b, d)


@pytest.mark.parametrize("gens", [40, 70])
def test_no_room_for_a_third_pair(gb, torch_cuda, gens):
    torch_cuda.cuda.empty_cache()
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, os.path.abspath(__file__), str(gens)], cwd=root, env=dict(os.environ, PYTHONPATH=root), capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]


if __name__ == "__main__":
    _child(int(sys.argv[1]))
