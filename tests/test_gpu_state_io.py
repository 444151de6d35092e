"""The state's way to the host: interior and face ghosts of every precision
form, in the slots' single-threaded and multi-threaded ranges, with the
halo's edges and corners left alone."""
import numpy as np
import pytest

from fall3d_b200 import ads
from fall3d_b200 import workloads as W
from fall3d_b200.ads import Domain

pytestmark = pytest.mark.gpu


# one slot; several slots, one thread; chunks that end inside a plane, four threads
@pytest.mark.parametrize("shape", [(5, 3, 2, 1), (61, 45, 31, 9), (233, 101, 23, 5)])
@pytest.mark.parametrize("prec", [ads.PREC_FP64, ads.PREC_FP32, ads.PREC_FP32C])
def test_download_places_every_row(built_lib, shape, prec):
    nx, ny, nz, nb = shape
    wl = W.small_case(nx, ny, nz, nb, seed=5)
    rng = np.random.default_rng(7)
    c0 = np.asfortranarray(rng.uniform(0.0, 1.0, (nx + 4, ny + 4, nz + 4, nb)))
    a0 = np.asfortranarray(rng.uniform(0.0, 1.0, (nx + 4, ny + 4, nb)))
    with Domain(wl.grid, nb, precision=prec) as dom:
        dom.upload_state(c0, a0)
        c = np.full_like(c0, -7.0, order="F")
        a = np.full_like(a0, -7.0, order="F")
        dom.download_state(c, a)
    x = c0[2:-2, 2:-2, 2:-2]
    if prec != ads.PREC_FP64:
        hi = x.astype(np.float32)
        x = hi.astype(np.float64) + ((x - hi).astype(np.float32) if prec == ads.PREC_FP32C else 0.0)
    want = np.full_like(c0, -7.0)
    want[2:-2, 2:-2, 2:-2] = x
    for h, e in ((0, 0), (1, 0), (-2, -1), (-1, -1)):
        want[h, 2:-2, 2:-2] = x[e]
        want[2:-2, h, 2:-2] = x[:, e]
        want[2:-2, 2:-2, h] = x[:, :, e]
    assert np.array_equal(c, want)
    want_a = np.full_like(a0, -7.0)
    want_a[2:-2, 2:-2] = a0[2:-2, 2:-2]
    assert np.array_equal(a, want_a)
