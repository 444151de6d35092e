"""FP64 steps over states whose values lie around the limits of the short
divisions (f3d_common.cuh: 2^-966, 2^-1010, the subnormal range), mixed with
ordinary ones in the same warp: bit-identical to the oracle."""
import numpy as np
import pytest

from fall3d_b200 import workloads as W
from tests.helpers import acum_interior, interior, run_pair
from tests.test_gpu_parity import _assert_bitwise

pytestmark = pytest.mark.gpu


# everything in the fringe; a fringe beside ordinary values; just above the limits
@pytest.mark.parametrize("low,high,ordinary", [(-1074, -880, 0.0), (-1074, -940, 0.3), (-990, -930, 0.1), (-1074, -1000, 0.0)])
@pytest.mark.parametrize("limiter,tm", [(1, 1), (2, 2), (3, 2)])
def test_values_around_the_limits(oracle_mod, built_lib, low, high, ordinary, limiter, tm):
    wl = W.small_case(37, 26, 14, 3, seed=8, limiter=limiter, time_marching=tm)
    wl.src_vals = 0.0 * wl.src_vals
    rng = np.random.default_rng(17)
    c0, a0 = W.random_state(wl, seed=5)
    shape = c0[2:-2, 2:-2, 2:-2].shape
    v = np.ldexp(rng.uniform(1.0, 2.0, shape), rng.integers(low, high, shape))
    v[rng.random(shape) < 0.1] = 0.0
    keep = rng.random(shape) < ordinary
    c0[2:-2, 2:-2, 2:-2] = np.where(keep, c0[2:-2, 2:-2, 2:-2], v)
    (c_o, a_o, _), (c_g, a_g, _), _ = run_pair(oracle_mod, wl, nsteps=3, dt=7.5, c0=c0, acum0=a0)
    _assert_bitwise(interior(c_o), interior(c_g), "c")
    _assert_bitwise(acum_interior(a_o), acum_interior(a_g), "acum")
