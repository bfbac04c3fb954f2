"""A host thread whose first CUDA call is one of the library's: every kind of call works, those that describe their
fields to the tensor memory accelerator (a driver call, which needs a current context) included."""
import ctypes
import threading

import pytest

from appfis_gb300 import _lib
from appfis_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _star(gb, torch, tile):
    f, w, ci = [torch.rand(152 * 56 * 58, device="cuda") for _ in range(2)], (ctypes.c_float * 5)(*W.fdtd_weights()), ctypes.c_int(-1)
    return f, lambda: gb.call("appfis_gb_star_r4", f[0].data_ptr(), f[1].data_ptr(), 0, 140, 48, 50, 152, 2, 1, 0.1, w, tile, 0, ctypes.byref(ci), None)


def _himeno(gb, torch, mixed):
    nx, ny, nz, pitch = 190, 180, 180, 192  # 6.2 M points: the TMA-staged sweeps
    f = [torch.rand(pitch * (ny + 2) * (nz + 2), device="cuda") * 0.1 for _ in range(14)]
    half, g, ci = torch.zeros(13 * f[0].numel(), dtype=torch.float16, device="cuda"), torch.zeros(3, dtype=torch.float64, device="cuda"), ctypes.c_int(-1)
    c = (ctypes.c_void_p * 12)(*[x.data_ptr() for x in f[2:]])
    if mixed:
        return f, lambda: gb.call("appfis_gb_himeno_mixed", c, f[0].data_ptr(), f[1].data_ptr(), half.data_ptr(), nx, ny, nz, pitch, 3, 3, 0.8,
                                  g.data_ptr(), ctypes.byref(ci), None)
    return f, lambda: gb.call("appfis_gb_himeno", c, f[0].data_ptr(), f[1].data_ptr(), nx, ny, nz, pitch, 3, 0.8, g.data_ptr(), ctypes.byref(ci), None)


def _heat(gb, torch):
    f, ci = [torch.rand(102 * 82, device="cuda") for _ in range(2)], ctypes.c_int(-1)
    return f, lambda: gb.call("appfis_gb_heat2d", f[0].data_ptr(), f[1].data_ptr(), 100, 80, 102, 20, 0.2, 0.2, ctypes.byref(ci), None)


def _life(gb, torch):
    f, ci = [(torch.rand(700 * 500, device="cuda") < 0.3).to(torch.uint8) for _ in range(2)], ctypes.c_int(-1)
    return f, lambda: gb.call("appfis_gb_life_u8", f[0].data_ptr(), f[1].data_ptr(), 700, 500, 9, 0, ctypes.byref(ci), None)


CALLS = {"star tma": lambda gb, t: _star(gb, t, 0), "star two steps": lambda gb, t: _star(gb, t, _lib.STAR_TB2),
         "himeno tma": lambda gb, t: _himeno(gb, t, False), "himeno mixed": lambda gb, t: _himeno(gb, t, True), "heat": _heat, "life": _life}


@pytest.mark.parametrize("name", CALLS)
def test_first_call(gb, torch_cuda, name):
    torch = torch_cuda
    torch.manual_seed(3)
    fields, call = CALLS[name](gb, torch)
    first = [f.clone() for f in fields]
    call()
    torch.cuda.synchronize()
    want = [f.clone() for f in fields]
    for f, v in zip(fields, first):
        f.copy_(v)
    torch.cuda.synchronize()
    raised = []

    def run():
        try:
            call()
        except Exception as e:  # noqa: BLE001  (reported below)
            raised.append(e)

    t = threading.Thread(target=run)
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert not raised, raised
    for f, v in zip(fields, want):
        assert torch.equal(f, v)


def test_flood_in_a_thread(gb, torch_cuda):
    doms, out = [W.triton_domain(60, 70, 3)], []
    args = (10.0, 0.5, 1e-3, 0.035, 600.0, 600.0, 1.0)
    want = _lib.flood_job(doms, *args, max_steps=6, dtype=_lib.F32)
    t = threading.Thread(target=lambda: out.append(_lib.flood_job(doms, *args, max_steps=6, dtype=_lib.F32)))
    t.start()
    t.join()
    assert len(out) == 1 and (out[0]["h"][0] == want["h"][0]).all()
