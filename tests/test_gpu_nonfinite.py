"""States with infinite, overflowing or NaN values: the CFL rate and the
operator answer as the oracle does (an infinite speed gives an infinite rate,
a NaN rate is passed over, a cell's bad value reaches the faces whose stencil
uses it and no others).  At fourth order products with metric factors that
vanish are not formed, so 0 * inf of the oracle (a NaN next to an overflowed
dissipation) is no NaN here; the cases keep to pressures, whose faces are the
same in both."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu

if gpu_available():
    import torch

    import heliocubed_b200 as hc
    from heliocubed_b200.level import make_box, wind_box_state

NR, NA = 20, 16


def _pair(po, **kw):
    if not gpu_available():
        pytest.skip("no CUDA device")
    kw = dict(dict(nr=NR, na=NA), **kw)
    return hc.Shell(hc.Params(**kw)), po.OracleLevel(po.make_params(**kw))


@pytest.mark.parametrize("component,value", [(4, np.inf), (4, -np.inf), (4, np.nan), (1, np.inf), (2, 1e200),
                                             (5, -np.inf), (6, 1e200), (0, np.nan)])
def test_cfl_rate_of_a_bad_cell(oracle_lib, component, value):
    """One bad cell in the first lane of a warp and in another lane: the rate
    is the oracle's (1e-13, or both infinite)."""
    sh, orc = _pair(oracle_lib)
    ju = sh.init_perturbed_wind(3)
    nv = NA * NA * NR
    for cell in (0, 64 + 21, 6 * nv - 1):
        bad = ju.clone()
        bad.view(6, 8, -1)[cell // nv, component, cell % nv] = value
        want, got = orc.inv_dt(bad.cpu().numpy()), sh.inv_dt_max(bad).item()
        same = got == want if np.isinf(want) else abs(got - want) <= 1e-13 * want
        assert same, (cell, got, want)


def test_time_step_beside_a_nan_cell():
    """The rate that a step leaves for the next one: the largest of the finite
    cells, also where a warp's first lane is a NaN cell (i = 0; the fastest
    cell is 12 cells further in the same row)."""
    if not gpu_available():
        pytest.skip("no CUDA device")
    sh = hc.Shell(hc.Params(nr=32, na=NA))
    first = sh.init_perturbed_wind(3)
    v = first.view(6, 8, NA, NA, 32)
    v[0, 4, 8, 8, 0] = np.nan
    v[0, 4, 8, 8, 12] *= 1e4
    one, two = first.clone(), first.clone()
    t1, t2 = (torch.zeros(1, dtype=torch.float64, device="cuda") for _ in range(2))
    sh.advance(one, 1, t1)
    sh.advance(two, 2, t2)
    rate = sh.inv_dt_max(one).item()
    assert one.view(6, 8, NA, NA, 32)[0, :, 8, 8, 0].isnan().any() and 0 < rate < np.inf
    dt = sh.params.cfl / rate
    assert abs((t2 - t1).item() - dt) <= 1e-10 * dt


def _assert_same(got, want):
    """Finite values in the same places, and there equal to 1e-12 of the
    component's largest."""
    got, want = got.reshape(8, -1), want.reshape(8, -1)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    for g, w in zip(got, want):
        m = np.isfinite(w)
        if m.any():
            assert np.abs(g[m] - w[m]).max() <= 1e-12 * np.abs(w[m]).max()


@pytest.mark.parametrize("riemann,component,value", [(1, 4, np.inf), (2, 4, np.inf), (2, 4, 1e200), (1, 6, 1e200),
                                                     (2, 6, -1e200)])
def test_operator_of_an_infinite_speed(oracle_lib, riemann, component, value):
    _check_level(oracle_lib, 3, riemann, component, value)


@pytest.mark.parametrize("limiter,riemann", [(0, 1), (1, 1), (2, 2), (3, 1), (3, 2)])
@pytest.mark.parametrize("component,value", [(0, np.nan), (1, np.nan), (3, -np.inf), (4, np.nan), (6, np.nan)])
def test_limiter_of_a_bad_cell(oracle_lib, limiter, riemann, component, value):
    _check_level(oracle_lib, limiter, riemann, component, value)


@pytest.mark.parametrize("limiter", [1, 3])
@pytest.mark.parametrize("value", [np.inf, -np.inf])
def test_limiter_of_an_infinity_in_a_flat_field(oracle_lib, limiter, value):
    """Differences 0 and infinity."""
    _check_level(oracle_lib, limiter, 1, 6, value, flat=True)


def _check_level(oracle_lib, limiter, riemann, component, value, flat=False):
    sh, orc = _pair(oracle_lib, limiter=limiter, riemann_solver=riemann)
    w = orc.prepare(sh.init_perturbed_wind(5).cpu().numpy(), 0.0)
    if flat:
        w.reshape(6, 8, -1)[:, component] = 0.0
    w.reshape(6, 8, NA + 4, NA + 4, NR + 4)[2, component, 7, 6, 9] = value
    got = sh.rhs(torch.from_numpy(w).cuda()).cpu().numpy()
    _assert_same(got.reshape(6, 8, -1).swapaxes(0, 1), orc.rhs(w).reshape(6, 8, -1).swapaxes(0, 1))


@pytest.mark.parametrize("riemann,fallback,component,value", [(1, 0, 4, np.inf), (1, 1, 4, np.inf), (2, 1, 4, np.inf),
                                                              (2, 0, 4, 1e200)])
def test_o4_operator_of_an_infinite_speed(oracle_lib, riemann, fallback, component, value):
    _check_o4_box(oracle_lib, riemann, fallback, component, value)


def _check_o4_box(oracle_lib, riemann, fallback, component, value):
    sh, orc = _pair(oracle_lib, spatial_order=4, riemann_solver=riemann, berta_fallback_type=fallback)
    lo, hi = (6, 4, 3), (11, 9, 10)
    v = [h - low + 1 for low, h in zip(lo, hi)]
    u = wind_box_state(sh.params, lo, hi, 5, seed=3)
    u.reshape(8, v[2] + 10, v[1] + 10, v[0] + 10)[component, 8, 7, 9] = value
    box = oracle_lib.HcBox()
    for d in range(3):
        box.lo[d], box.hi[d] = lo[d], hi[d]
    box.ghost, box.block = 5, 1
    want = np.zeros(8 * int(np.prod(v)))
    orc.box_rhs_o4(box, u, want)
    got = torch.zeros(want.size, dtype=torch.float64, device="cuda")
    sh.box_rhs_o4(make_box(lo, hi, 5, 1), torch.from_numpy(u).cuda(), got)
    _assert_same(got.cpu().numpy(), want)


@pytest.mark.parametrize("riemann,fallback", [(1, 0), (2, 0), (1, 1), (2, 1)])
def test_o4_operator_of_an_infinite_density(oracle_lib, riemann, fallback):
    """The cell is at rest: its finite momenta over the density are 0."""
    _check_o4_box(oracle_lib, riemann, fallback, 0, np.inf)


def test_primitives_of_an_infinite_density(oracle_lib):
    sh, orc = _pair(oracle_lib)
    ju = sh.init_perturbed_wind(5)
    ju.view(6, 8, NA, NA, NR)[3, 0, 7, 5, 9] = np.inf
    cell = (3, slice(None), 9, 7, 11)  # two ghosts
    got, want = (w.reshape(6, 8, NA + 4, NA + 4, NR + 4)[cell]
                 for w in (sh.prepare(ju).cpu().numpy(), orc.prepare(ju.cpu().numpy(), 0.0)))
    assert np.array_equal(got[1:4], np.zeros(3)) and np.array_equal(np.isfinite(got), np.isfinite(want))
