"""A box whose rows are nearly 2^31 elements long (17 GB): positions past a row's end are still found in the next."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("code", [0, 2])
def test_rows_of_nearly_2_31(gb, torch_cuda, code):
    torch = torch_cuda
    px, skip = 2 ** 31 - 1, 1000
    if torch.cuda.mem_get_info()[0] < 20 << 30:
        pytest.skip("needs 20 GB of device memory")
    dt = torch.float32 if code == 0 else torch.int32
    f = torch.ones((2, px), dtype=dt, device="cuda")
    f[:, px - skip:] = 7  # not in the box
    f[1, :3] = 4
    out = torch.zeros(1, dtype=torch.float64 if code == 0 else torch.int64, device="cuda")
    box = (ctypes.c_int * 6)(0, px - skip, 0, 2, 0, 1)
    got = []
    for op in (0, 1, 2):
        gb.call("appfis_gb_reduce", f.data_ptr(), code, px, 2, box, op, out.data_ptr(), None)
        gb.call("appfis_gb_stream_sync", None)
        got.append(out.item())
    del f
    torch.cuda.empty_cache()
    assert got == [4, 1, 2 * (px - skip) + 9]
