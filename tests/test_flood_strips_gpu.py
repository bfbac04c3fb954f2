"""Strip heights of the flood passes: a domain's fields, step count and time steps do not depend on the
batch it runs in, whose size sets the rows per strip (2 alone; 4, 8 or 16 beside a larger domain).
Heights, widths and last strips cut at odd places; bit for bit, as strips only share out the cells."""
import numpy as np
import pytest

from appfis_gb300 import _lib
from appfis_gb300 import workloads as W

pytestmark = pytest.mark.gpu
ARGS = (10.0, 0.5, 1e-3, 0.035, 600.0, 600.0, 1.0)
STEPS = 24


def _small():
    return [W.triton_domain(ny, nx, 700 + nx) for ny, nx in ((37, 130), (3, 5), (97, 56), (66, 29))]


@pytest.mark.parametrize("flags", [0, _lib.FLOOD_SKIP_DRY, _lib.FLOOD_TWO_PHASE, _lib.FLOOD_UNSTAGED])
@pytest.mark.parametrize("dtype,beside", [(_lib.F32, 620), (_lib.F32, 1950), (_lib.F32, 3750), (_lib.F64, 1950), (_lib.F64, 3100)])
def test_fields_do_not_depend_on_the_batch(gb, torch_cuda, dtype, beside, flags):
    if dtype == _lib.F64 and flags == _lib.FLOOD_UNSTAGED:
        pytest.skip("FP64 rows are never staged")
    doms = _small()
    alone = _lib.flood_job(doms, *ARGS, max_steps=STEPS, dtype=dtype, flags=flags)
    flat = (np.zeros((beside, beside)), np.zeros((beside, beside)))
    flat[1][10:20, 10:20] = 0.5
    batch = _lib.flood_job(doms + [flat], *ARGS, max_steps=STEPS, dtype=dtype, flags=flags)
    for k in range(len(doms)):
        assert batch["steps"][k] == alone["steps"][k]
        assert np.array_equal(batch["dts"][k], alone["dts"][k])
        for f in ("h", "qx", "qy"):
            assert np.array_equal(batch[f][k], alone[f][k]), (k, f)
    assert all(h.any() for h in batch["h"])
