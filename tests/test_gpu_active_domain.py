"""A Domain's sweeps over the non-zero boxes (active.cuh) against the same
Domain marching every cell, bit for bit.

An empty last bin with a settling velocity beyond the bound of a calm field
makes every cell count and touches nothing else.  Uploading a state makes the
next step look for its boxes whatever the last ones gained (box_gate.h), so
the state goes through the host before every step or operator."""
import numpy as np
import pytest

from fall3d_b200 import workloads as W
from fall3d_b200.ads import PREC_FP32, PREC_FP32C, Domain
from fall3d_b200.ensemble import MODE_KERNELS, MODE_PERSISTENT, Ensemble
from tests.test_gpu_active import _puffs

pytestmark = pytest.mark.gpu

NB = 3
DT = 30.0


def _bits(a):
    """Values by their bits, NaN as one value."""
    a = np.where(np.isnan(a), np.nan, a)
    return a.view(np.int64)


def _pair(shape, prec, lim=2, tm=2, nb=NB, seed=11):
    """The boxed domain and the one that marches every cell, and their workload."""
    wl = W.small_case(*shape, nb, seed=seed)
    g = wl.grid
    vs = np.zeros((g.nx, g.ny, g.nz + 3, nb), order="F")
    vs += np.linspace(2.0, 0.01, nb) * np.linspace(1.0, 1.2, g.nz + 3)[:, None]
    doms = []
    for wild in (False, True):
        v = vs.copy(order="F")
        if wild:
            v[0, 0, :, nb - 1] = 2e12
        dom = Domain(g, nb, lim, tm, prec)
        dom.set_meteo(wl.u12, wl.v12, wl.w12, wl.k1, wl.k2, wl.k3, v, wl.t_its, wl.t_ite)
        dom.keep_boundary_halo(True)
        doms.append(dom)
    return wl, doms


def _zeros(g, nb):
    return np.zeros((g.nx + 4, g.ny + 4, g.nz + 4, nb), order="F"), np.zeros((g.nx + 4, g.ny + 4, nb), order="F")


def _same(states):
    """The same bits inside; ghosts and sums of nothing but zeros may differ in the zero's sign."""
    for a, b in zip(*states):
        assert np.array_equal(a, b, equal_nan=True)
        if a.ndim == 4:
            assert np.array_equal(_bits(a[2:-2, 2:-2, 2:-2]), _bits(b[2:-2, 2:-2, 2:-2]))


def _steps(doms, c0, a0, times, extra=lambda d: []):
    out = []
    for d in doms:
        c, a, f = c0.copy(order="F"), a0.copy(order="F"), np.zeros(6)
        for it, t in enumerate(times):
            d.upload_state(c, a)
            d.F3D_time_step(DT, t, it, f)
            c, a = d.download_state(c, a)
        out.append([c, a] + extra(d))
        assert np.isfinite(f).all() or np.isnan(c).any()
    return out


# rows longer than a chunk of the scan, tiles of every raggedness; both orders of x and y
@pytest.mark.parametrize("shape", [(300, 21, 9), (70, 41, 33), (17, 300, 6)])
@pytest.mark.parametrize("prec,lim,tm", [(PREC_FP32, 1, 2), (PREC_FP32, 2, 1), (PREC_FP32C, 2, 2), (PREC_FP32C, 3, 1)])
@pytest.mark.parametrize("where", [[(0.5, 0.5, 0.5)], [(0, 0, 0), (1, 1, 1)], []])
def test_steps(built_lib, shape, prec, lim, tm, where):
    wl, doms = _pair(shape, prec, lim, tm)
    c0, a0 = _puffs(wl, where), _zeros(wl.grid, NB)[1]
    vals = np.array(wl.src_vals, dtype=np.float64).reshape(-1, NB)
    vals[:, NB - 1] = 0.0
    for d in doms:
        d.set_source(wl.src_ijk, vals)  # in levels that are empty, too
    out = _steps(doms, c0, a0, [100.0, 130.0, 160.0])
    _same(out)
    assert (out[0][0] != 0).any()


@pytest.mark.parametrize("prec", [PREC_FP32, PREC_FP32C])
@pytest.mark.parametrize("where", [[(0.5, 0.5, 0.5)], [(0.02, 0.9, 0.1), (0.9, 0.2, 0.8)]])
def test_operators_one_by_one(built_lib, prec, where):
    wl, doms = _pair((130, 75, 14), prec)
    c0, a0 = _puffs(wl, where), _zeros(wl.grid, NB)[1]
    out = []
    for d in doms:
        c, a, fl = c0.copy(order="F"), a0.copy(order="F"), []
        for turn in ("xyz", "yxz", "zyx"):
            d.ADS_update_horizontal_vcomps(0.3)
            for q in turn:
                d.upload_state(c, a)
                fl += {"x": lambda: d.ADS_solve_along_x(DT), "y": lambda: d.ADS_solve_along_y(DT),
                       "z": lambda: d.ADS_solve_along_z(DT, 0.3)}[q]()
                c, a = d.download_state(c, a)
        out.append([c, a, np.array(fl)])
    _same(out)


@pytest.mark.parametrize("prec", [PREC_FP32, PREC_FP32C])
def test_wet_deposition_and_decay(built_lib, prec):
    from tests.test_gpu_wetdep import A, B, CAT, DIAM, SPE
    nb = len(CAT)
    wl, doms = _pair((90, 60, 20), prec, nb=nb)
    g, rng = wl.grid, np.random.default_rng(2)
    pre = np.asfortranarray(rng.uniform(0.0, 30.0, (g.nx, g.ny)))
    pblh = np.asfortranarray(rng.uniform(300.0, 2500.0, (g.nx, g.ny)))
    c0, a0 = _zeros(g, nb)
    c0[40:44, 30:33, 5:9, :nb - 1] = rng.uniform(1e-6, 1e-3, (4, 3, 4, nb - 1))
    for d in doms:
        d.phys_wet_deposition(A, B, pre, pblh, CAT, DIAM)
        d.phys_radionuclides(CAT, SPE)
    _same(_steps(doms, c0, a0, [0.0, 30.0, 60.0], lambda d: [d.get_awet()]))


@pytest.mark.parametrize("prec", [PREC_FP32, PREC_FP32C])
def test_gravity_current_on_and_off(built_lib, prec):
    wl, doms = _pair((60, 50, 12), prec)
    g = wl.grid
    c0, a0 = _puffs(wl, [(0.3, 0.4, 0.5)]), _zeros(g, NB)[1]
    for d in doms:
        d.set_gravity_current(g.lon_c[13], g.lat_p[9], 40.0, 110.0, 430.0, 0.1, 0.02, 0.2, 1e7, 3000.0, 0.0)
    _same(_steps(doms, c0, a0, [30.0 * q for q in range(6)]))


@pytest.mark.parametrize("prec", [PREC_FP32, PREC_FP32C])
@pytest.mark.parametrize("value", [-0.0, np.nan, np.inf, 1e-45])
def test_odd_values_in_the_state(built_lib, prec, value):
    wl, doms = _pair((90, 40, 12), prec)
    c0, a0 = _zeros(wl.grid, NB)
    c0[50, 20, 7, 0] = value
    c0[10, 30, 4, 1] = 1e-4
    out = _steps(doms, c0, a0, [0.0, 30.0])
    _same(out)
    if not np.isfinite(value):
        assert np.isnan(out[0][0][..., 0]).any() and np.isfinite(out[0][0][..., 1]).all()


def test_an_infinite_wind_far_from_the_ash_counts(built_lib):
    """0 times an infinite wind is NaN wherever the ash is: the per-phase
    kernels must march there as the persistent kernel does, and march over the
    boxes again once the field is finite."""
    wl = W.small_case(80, 40, 9, NB, seed=5)
    g = wl.grid
    u = wl.u12.copy(order="F")
    u[60, 30, 4, :] = np.inf
    vs = np.full((g.nx, g.ny, g.nz + 3, NB), 0.5, order="F")
    c0 = _puffs(wl, [(0.1, 0.1, 0.5)])
    out = []
    for mode, bpb in ((MODE_KERNELS, 4), (MODE_PERSISTENT, 2)):
        ens = Ensemble([g], NB, [0], [1.0], 2, 2, PREC_FP32C)
        ens.set_tuning(mode, bpb, 0)
        got = []
        for winds in (u, wl.u12):
            ens.set_class_meteo(0, winds, wl.v12, wl.w12, wl.k1, wl.k2, wl.k3, vs, wl.t_its, wl.t_ite)
            ens.upload_member_state(0, c0, None)
            ens.step(DT, 0.5 * (wl.t_its + wl.t_ite), 0)
            got.append(ens.download_member_state(0)[0])
        assert ens.status() == 0
        ens.close()
        out.append(got)
    assert np.isnan(out[0][0]).any() and np.isfinite(out[0][1]).all()
    _same(out)


@pytest.mark.parametrize("prec", [PREC_FP32, PREC_FP32C])
def test_boxes_are_looked_for_where_they_pay(built_lib, prec):
    """Two launches more a step while a puff leaves most of a long domain
    empty; none once ash is everywhere, but for a look now and then; the same
    on the way back."""
    wl, (dom, _) = _pair((400, 24, 8), prec)
    puff = _puffs(wl, [(0.5, 0.5, 0.5)])
    full, a0 = _zeros(wl.grid, NB)
    full[2:-2, 2:-2, 2:-2] = 1e-4

    def launches(n):
        got = []
        for it in range(n):
            before = dom.launch_count()
            dom.F3D_time_step(1.0, 0.0, it, np.zeros(6))
            got.append(dom.launch_count() - before)
        return got
    dom.upload_state(puff, a0)
    with_boxes = launches(5)
    assert len(set(with_boxes)) == 1
    dom.upload_state(full, a0)
    dense = launches(40)
    plain = with_boxes[0] - 2
    assert dense[0] == with_boxes[0] and set(dense) == {plain, plain + 2} and dense.count(plain + 2) <= 4
    dom.upload_state(puff, a0)
    assert launches(5) == with_boxes
