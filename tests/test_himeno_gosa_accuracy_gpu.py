"""gosa of the flat Himeno sweep as accurate as a sum in doubles.  With every neighbour coefficient 0, a3 = bnd = 1 and
p = 0 a point's ss is its wrk1, so the test chooses the squares; rows of 62 points at a pitch of 64 put the same 31
values in every other warp, whose sum in two floats is off by 2^-46.5, each time the same way."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NX, NY, NZ, PITCH = 62, 62, 64, 64
VALUES = [0x4022f1a6, 0x3fc5de84, 0x3f8042af, 0x4306ea2f, 0x3e5c4f25, 0x3df68003, 0x3fc194ad, 0x3e9b012c,
          0x3fe61b3d, 0x3f965c90, 0x3f791ed9, 0x3fd73e41, 0x3eaae980, 0x3ddd990f, 0x3f39fcde, 0x3e03b401,
          0x408bb9e6, 0x40292da4, 0x3f2f21dc, 0x3fac7740, 0x3e6cbe4c, 0x41ac35d7, 0x41087ca3, 0x3de4a4ff,
          0x4090aba1, 0x40508916, 0x3ecf6336, 0x401d0340, 0x3e2f3797, 0x3ff29191, 0x3fb6bc88, 0x4127479c,
          0x41050900, 0x3f309aef, 0x3fa53b3f, 0x410507fe, 0x3eea10d6, 0x4106d2e4, 0x40f70ef1, 0x3fe731cb,
          0x3f7fa19a, 0x40fb5a3a, 0x3f2ad70e, 0x3eb801fc, 0x401950c1, 0x40f01ac3, 0x3f595299, 0x404da1ea,
          0x4044135e, 0x3fe2c3fc, 0x3fc77afa, 0x3d0478c6, 0x3fb1a6f7, 0x3f13cd78, 0x3f5ce456, 0x3fba233a,
          0x3f346dc3, 0x3f9e4c08, 0x3f34e4db, 0x40172d01, 0x3f99cc31, 0x400e4335]


def _gosa(gb, torch, row):
    """One sweep over a grid whose odd planes have `row` in every row of wrk1, so a thread (2 planes) has one term."""
    wrk1 = torch.zeros((NZ + 2, NY + 2, PITCH), dtype=torch.float32, device="cuda")
    wrk1[1:NZ:2, 1:NY + 1, 1:NX + 1] = torch.from_numpy(row).cuda()
    zero, one = torch.zeros_like(wrk1), torch.ones_like(wrk1)
    fields = [zero, zero, zero, one, zero, zero, zero, zero, zero, zero, one, wrk1]  # a0-a3 b0-b2 c0-c2 bnd wrk1
    a, b = torch.zeros_like(wrk1), torch.zeros_like(wrk1)
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    gb.call("appfis_gb_himeno", (ctypes.c_void_p * 12)(*[f.data_ptr() for f in fields]), a.data_ptr(), b.data_ptr(), NX, NY, NZ, PITCH, 1, 0.8,
            out.data_ptr(), None, None)
    gb.call("appfis_gb_stream_sync", None)
    return out.item()


def test_values_that_two_floats_lose(gb, torch_cuda):
    row = np.array(VALUES, dtype=np.uint32).view(np.float32)
    exact = math.fsum(row.astype(np.float64) ** 2) * NY * (NZ // 2)  # a float's square is exact in a double
    # roundings of a sum in doubles: a warp's sum 1 (5 as doubles), the block's 3, of 512 block sums 2 per thread, then 5 and 8
    assert abs(_gosa(gb, torch_cuda, row) - exact) <= 23 * 2.0 ** -53 * exact


def test_warp_sums_beyond_the_float_range(gb, torch_cuda):
    row = np.full(NX, 1e19, dtype=np.float32)  # a square is 1e38, a warp's sum 3e39
    exact = float(row[0]) ** 2 * NX * NY * (NZ // 2)
    assert abs(_gosa(gb, torch_cuda, row) - exact) <= 23 * 2.0 ** -53 * exact
    row[5] = np.inf
    assert not math.isfinite(_gosa(gb, torch_cuda, row))
