"""Read-backs before and after a context has moved enough for the larger slots."""
import numpy as np
import pytest

from fall3d_b200 import ads
from fall3d_b200 import workloads as W
from fall3d_b200.ads import Domain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [ads.PREC_FP64, ads.PREC_FP32C])
def test_many_read_backs(built_lib, prec):
    nx, ny, nz, nb = 233, 101, 23, 5  # 21.6 MB of values, rows that do not fill a slot
    wl = W.small_case(nx, ny, nz, nb, seed=5)
    rng = np.random.default_rng(7)
    c0 = np.asfortranarray(rng.uniform(0.0, 1.0, (nx + 4, ny + 4, nz + 4, nb)))
    x = c0[2:-2, 2:-2, 2:-2]
    if prec != ads.PREC_FP64:
        hi = x.astype(np.float32)
        x = hi.astype(np.float64) + (x - hi).astype(np.float32)
    with Domain(wl.grid, nb, precision=prec) as dom:
        dom.upload_state(c0, None)
        c = np.empty_like(c0)
        for _ in range(21):  # past the 128 MB that bring them
            c.fill(-7.0)
            dom.download_state(c, None)
            assert np.array_equal(c[2:-2, 2:-2, 2:-2], x)
