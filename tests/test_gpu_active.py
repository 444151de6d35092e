"""Sweeps over the non-zero boxes (active.cuh) against sweeps over every cell.

The persistent step kernel marches over whole pencils, the per-phase kernels
over the boxes; a state of isolated puffs must come out of both the same, bit
for bit, as must one whose winds are not bounded (every cell then counts)."""
import numpy as np
import pytest

from fall3d_b200 import workloads as W
from fall3d_b200.ensemble import MODE_KERNELS, MODE_PERSISTENT, Ensemble

pytestmark = pytest.mark.gpu

NB = 3


def _puffs(wl, where):
    """Halo-inclusive state: one cell or small cube per bin and place, nothing in the last bin."""
    g = wl.grid
    c = np.zeros((g.nx + 4, g.ny + 4, g.nz + 4, NB), order="F")
    rng = np.random.default_rng(3)
    for b in range(NB - 1):
        for (fx, fy, fz) in where:
            i, j, k = (2 + int(f * (n - 1)) for f, n in ((fx, g.nx), (fy, g.ny), (fz, g.nz)))
            c[i:min(i + 1 + b, g.nx + 2), j, k, b] = rng.uniform(1e-6, 1e-3)
    return c


def _run(wls, states, mode, prec, lim, tm):
    ens = Ensemble([w.grid for w in wls], NB, list(range(len(wls))), [1.1] * len(wls), lim, tm, prec)
    ens.set_tuning(mode, 4 if mode == MODE_KERNELS else 2, 0)
    ens.keep_boundary_halo(True)
    for q, w in enumerate(wls):
        ens.set_class_meteo(q, w.u12, w.v12, w.w12, w.k1, w.k2, w.k3, w.vs, w.t_its, w.t_ite)
        ens.upload_member_state(q, states[q], None)
    ens.compute_time_steps(0.5, 2, 0.9, 20.0)
    ens.set_clock(np.zeros(len(wls)), 0)
    ens.run(3)
    out = [ens.download_member_state(q) for q in range(len(wls))]
    fl = ens.get_fluxes()
    assert ens.status() == 0
    ens.close()
    return out, fl


# a pencil shorter than a box's reach, ragged tiles, rows longer than a chunk of the staging
@pytest.mark.parametrize("prec,lim,tm", [(1, 1, 2), (1, 2, 1), (2, 2, 2), (2, 3, 2), (2, 1, 1)])
@pytest.mark.parametrize("where", [[(0.5, 0.5, 0.5)], [(0, 0, 0), (1, 1, 1)], [(0.1, 0.9, 0.2), (0.15, 0.2, 0.2)], []])
@pytest.mark.parametrize("wild", [False, True])
def test_boxes_change_no_bit(built_lib, prec, lim, tm, where, wild):
    wls = [W.small_case(*s, NB, seed=11 + q) for q, s in enumerate([(70, 41, 33), (9, 67, 12), (33, 7, 5)])]
    if wild:  # beyond the bound of a calm field, still finite
        for w in wls:
            w.k1 = w.k1.copy(order="F")
            w.k1[2, 0, 0] = 2e12
    states = [_puffs(w, where) for w in wls]
    (a, fa), (b, fb) = (_run(wls, states, mode, prec, lim, tm) for mode in (MODE_KERNELS, MODE_PERSISTENT))
    for (ca, aa), (cb, ab) in zip(a, b):
        assert np.array_equal(ca, cb, equal_nan=True)
        assert np.array_equal(aa, ab, equal_nan=True)
    assert np.allclose(fa, fb, rtol=1e-12, atol=0, equal_nan=True)
