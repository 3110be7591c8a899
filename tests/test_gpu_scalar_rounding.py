"""Rounding of the scalar assembly against extended precision, on edges that
share no node, so that a row holds one edge's entries; below and above the
edge count where the node pre-pass starts.

* tanh Peclet function near one: the downwind entry is mdot / 2 (1 - pec) and
  1 - pec = 1 / (1 + exp(2 y)), y = (pe - trans) / width. Its relative error is
  2 |dy| plus a few units: pe <= 140 comes from about eight roundings
  (2 * 8 * 140 / 4 = 560 units) and each other factor from one, so 1,024 units
  bound it. Formed as 1 - pec it would keep no digit beyond 2^-53 of one.
* the relaxed diagonal is the opposite entry over the relaxation factor,
  rounded once."""
import numpy as np
import pytest

from gpu_util import scalar_fields, to_dev_dict

pytestmark = pytest.mark.gpu


def _pairs(nw, E, seed, od, area, pe):
    """E disjoint edges with Peclet numbers pe, positive mass flow."""
    rng = np.random.default_rng(seed)
    N = 2 * E
    edges = np.arange(N, dtype=np.int64).reshape(E, 2)
    coords = rng.uniform(size=(N, 3))
    coords[1::2] = coords[::2] + rng.uniform(0.5, 1.0, size=(E, 3))
    vel = rng.uniform(0.5, 1.0, size=(N, 3))
    rho = rng.uniform(0.8, 1.2, N)
    dx = coords[1::2] - coords[::2]
    udx = 0.5 * np.sum(dx * (vel[1::2] + vel[::2]), 1)
    diff = np.repeat(udx / pe, 2) * rho
    f = dict(coords=coords, velocity=vel, q=rng.uniform(size=N), dqdx=rng.normal(size=(N, 3)), density=rho, diff=diff,
             area=area * dx * rng.uniform(0.9, 1.1, size=(E, 3)), mdot=rng.uniform(0.5, 1.5, E))
    ls = nw.LinearSystem(1)
    ls.build_edge_graph(N, edges)
    ls.finalize()
    ls.zero_system()
    ls.assemble_scalar(scalar_fields(nw, to_dev_dict(f)), nw.ScalarOpts(**od))
    v, _ = ls.to_host()
    v = v.reshape(E, 2, 2)
    return f, v


OPTS = dict(alpha=0.0, alpha_upw=1.0, upw_factor=1.0, hybrid_factor=1.0, use_limiter=1, tanh_trans=2.0, tanh_width=4.0)


@pytest.mark.parametrize("E", [700, 131200])
def test_downwind_entry_near_full_upwinding(nw, E):
    od = dict(OPTS, relax=1.0, tanh_form=1)
    f, v = _pairs(nw, E, 1, od, 1e-60, np.linspace(42.0, 138.0, E))
    X = {k: a.astype(np.longdouble) for k, a in f.items()}
    dx = X["coords"][1::2] - X["coords"][::2]
    udx = np.sum(dx * (X["velocity"][1::2] + X["velocity"][::2]), 1) / 2
    d = X["diff"] / X["density"]
    pe = udx / ((d[::2] + d[1::2]) / 2 + np.longdouble(1e-16))
    om = 1 / (1 + np.exp(2 * (pe - 2) / 4))
    lf = -(X["diff"][::2] + X["diff"][1::2]) / 2 * np.sum(X["area"] ** 2, 1) / np.sum(X["area"] * dx, 1)
    ref = lf + X["mdot"] / 2 * om
    assert om.max() < 3e-9 and np.abs(lf / ref).max() < 1e-20
    err = np.abs(v[:, 0, 1] - ref) / np.abs(ref)
    assert err.max() <= 1024 * 2.0 ** -52, float(err.max())


@pytest.mark.parametrize("tanh_form", [0, 1])
@pytest.mark.parametrize("E", [700, 131200])
def test_relaxed_diagonal_is_rounded_once(nw, E, tanh_form):
    relax = 0.7
    f, v = _pairs(nw, E, 2, dict(OPTS, relax=relax, tanh_form=tanh_form), 1.0, np.geomspace(1e-3, 1e3, E))
    for diag, opposite in ((v[:, 0, 0], v[:, 1, 0]), (v[:, 1, 1], v[:, 0, 1])):
        err = np.abs(diag.astype(np.longdouble) + opposite.astype(np.longdouble) / np.longdouble(relax))
        assert np.all(err <= np.spacing(np.abs(diag)) * np.longdouble(0.5 + 2.0 ** -9))


def test_tanh_form_far_below_its_transition(nw):
    """exp(-2 y) beyond the FP64 range: pec is zero and the advection central."""
    od = dict(OPTS, relax=1.0, tanh_form=1, tanh_width=1e-3)
    f, v = _pairs(nw, 300, 3, od, 1e-60, np.full(300, 0.5))
    np.testing.assert_allclose(v[:, 0, 1], f["mdot"] / 2, rtol=1e-14)
    np.testing.assert_allclose(v[:, 1, 0], -f["mdot"] / 2, rtol=1e-14)
