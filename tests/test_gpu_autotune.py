"""The autotuner runs its candidates there and back, so that a plume that
grows while they are timed weighs on all of them alike."""
import numpy as np
import pytest

from fall3d_b200 import workloads as W
from fall3d_b200.ensemble import CANDIDATES, Ensemble, autotune

pytestmark = pytest.mark.gpu


def test_every_candidate_runs_twice(built_lib):
    wl = W.small_case(26, 18, 12, 3, seed=4)
    ens = Ensemble([wl.grid], 3, [0, 0], [1.0, 1.1], 2, 2, 2)
    ens.set_class_meteo(0, wl.u12, wl.v12, wl.w12, wl.k1, wl.k2, wl.k3, None, wl.t_its, wl.t_ite)
    ens.compute_class_vset(0, wl.vset_model, wl.rhoc, wl.tc, wl.diam, wl.rhop, wl.psi, wl.bin_cat)
    for m in range(2):
        ens.set_member_source(m, wl.src_ijk, wl.src_vals)
    dt = ens.compute_time_steps(0.5, 2, 0.9, 1e30)
    ens.set_clock(np.zeros(2), 0)
    best = autotune(ens, "unused", steps=3, use_cache=False)
    assert all(r.get("ms_per_step", 0.0) > 0.0 for r in best["all"])
    t = ens.get_clock()[0]
    assert np.allclose(t, 2 * CANDIDATES * (2 + 3) * dt, rtol=1e-12, atol=0)
    ens.close()
