"""f3d_ads_set_meteo_corners_kdiffu, the C entry that takes both time levels of
a corner field in one array, against f3d_ads_set_meteo_pairs_kdiffu (what
Domain calls): the same time step and state, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from fall3d_b200._lib import F3DKdiffu, check, lib
from fall3d_b200.ads import PREC_FP64, Domain, _p
from tests.test_gpu_kdiffu import NB, _run
from tests.test_kdiffu_ref import kdiffu_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("modkh,modkv,with_tvc", [(2, 3, True), (4, 1, True), (2, 1, False)])
def test_one_array_for_both_levels(built_lib, modkh, modkv, with_tvc):
    g, uc2, vc2, tvc2, pblh, mon, ust = kdiffu_case(22, 17, 10, seed=5)
    rng = np.random.default_rng(1)
    wc2 = [np.asfortranarray(rng.uniform(-0.4, 0.4, uc2[0].shape)) for _ in range(2)]
    c0 = np.zeros((g.nx + 4, g.ny + 4, g.nz + 4, NB), order="F")
    c0[2:-2, 2:-2, 2:-2] = rng.uniform(0, 1e-3, (g.nx, g.ny, g.nz, NB))
    got = []
    for joined in (False, True):
        dom = Domain(g, NB, precision=PREC_FP64)
        dom.set_terrain()
        if joined:
            dom._ensure_corner_heights()
            both = [np.asfortranarray(np.stack(f, axis=3)) for f in (uc2, vc2, wc2, tvc2)]
            if not with_tvc:
                both[3] = None
            two = [np.asfortranarray(f, dtype=np.float64) for f in (pblh, mon, ust, g.h_c)]
            kd = F3DKdiffu(modkh, modkv, int(g.map_h), 2500.0, 40.0, 0.2275, float(g.dlon), float(g.dlat), 0.25)
            check(lib().f3d_ads_set_meteo_corners_kdiffu(dom._h, *[_p(f) for f in both], *[_p(f) for f in two],
                                                         C.byref(kd), 0.0, 3600.0), "f3d_ads_set_meteo_corners_kdiffu")
        else:
            dom.set_meteo_corners_kdiffu(uc2, vc2, wc2, modkh, modkv, 0.25, tvc_pair=tvc2 if with_tvc else None,
                                         pblh=pblh, mon=mon, ust=ust, kh0=2500.0, kv0=40.0, t_its=0.0, t_ite=3600.0)
        got.append(_run(dom, g, c0))
        dom.close()
    assert got[0][0] == got[1][0]
    assert np.array_equal(got[0][1], got[1][1])
