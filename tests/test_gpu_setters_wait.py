"""A state that is uploaded while steps are in flight is the state afterwards:
the upload waits for them, and they do not run on over it."""
import numpy as np
import pytest

from fall3d_b200 import ads
from fall3d_b200 import workloads as W
from fall3d_b200.ads import Domain
from fall3d_b200.ensemble import Ensemble

pytestmark = pytest.mark.gpu

NB = 3


def _case():
    wl = W.small_case(120, 90, 30, NB, seed=3)
    g = wl.grid
    vs = np.full((g.nx, g.ny, g.nz + 3, NB), 0.5, order="F")
    rng = np.random.default_rng(4)
    a, b = (np.asfortranarray(rng.uniform(1e-6, 1e-3, (g.nx + 4, g.ny + 4, g.nz + 4, NB)).astype(np.float32)
                              .astype(np.float64)) for _ in range(2))
    return wl, vs, a, b


@pytest.mark.parametrize("prec", [ads.PREC_FP64, ads.PREC_FP32, ads.PREC_FP32C])
def test_domain(built_lib, prec):
    wl, vs, a, b = _case()
    with Domain(wl.grid, NB, precision=prec) as dom:
        dom.set_meteo(wl.u12, wl.v12, wl.w12, wl.k1, wl.k2, wl.k3, vs, wl.t_its, wl.t_ite)
        dom.upload_state(a, None)
        for it in range(200):
            dom.step_async(10.0, 100.0, it)
        dom.upload_state(b, None)
        got = dom.download_state()[0]
    assert np.array_equal(got[2:-2, 2:-2, 2:-2], b[2:-2, 2:-2, 2:-2])


@pytest.mark.parametrize("prec", [ads.PREC_FP64, ads.PREC_FP32C])
def test_ensemble(built_lib, prec):
    wl, vs, a, b = _case()
    ens = Ensemble([wl.grid], NB, [0, 0], [1.0, 1.1], 2, 2, prec)
    ens.set_class_meteo(0, wl.u12, wl.v12, wl.w12, wl.k1, wl.k2, wl.k3, vs, wl.t_its, wl.t_ite)
    for m in range(2):
        ens.upload_member_state(m, a, None)
    ens.compute_time_steps(0.5, 2, 0.9, 20.0)
    ens.set_clock(np.zeros(2), 0)
    ens.run(200)
    ens.upload_member_state(1, b, None)
    got = ens.download_member_state(1)[0]
    ens.close()
    assert np.array_equal(got[2:-2, 2:-2, 2:-2], b[2:-2, 2:-2, 2:-2])
