"""Systems below and above the sizes from which a node pre-pass is launched
(131,072 edges scalar, 262,144 continuity), against the oracle with the
tolerances of the parity tests."""
import numpy as np
import pytest

from gpu_util import check_close, continuity_fields, oracle_continuity, oracle_scalar, scalar_fields, to_dev_dict

pytestmark = pytest.mark.gpu


def _linsys(nw, N, edges):
    ls = nw.LinearSystem(1)
    ls.build_edge_graph(N, edges)
    ls.finalize()
    ls.zero_system()
    return ls


@pytest.mark.parametrize("noc", [1.0, 0.4])
@pytest.mark.parametrize("dims", [(1, 1, 1), (43, 43, 43), (44, 44, 44)])
def test_continuity(nw, orc, dims, noc):
    mesh = nw.Mesh(*dims, jitter=0.04, seed=4)
    assert (mesh.num_edges > 262144) == (dims[0] == 44)
    rng = np.random.default_rng(5)
    N = mesh.num_nodes
    f = dict(coords=mesh.coords, velocity=rng.normal(size=(N, 3)), dpdx=rng.normal(size=(N, 3)),
             density=rng.uniform(0.5, 2, N), pressure=rng.normal(size=N), udiag=rng.uniform(1, 3, N),
             area=mesh.area)
    od = dict(noc_fac=noc, tau_scale=0.5, interp_together=1.0, solve_incompressible=0.0)
    ref = oracle_continuity(orc, mesh.edges, mesh.nalu_id, f, od)
    ls = _linsys(nw, N, mesh.edges)
    ls.assemble_continuity(continuity_fields(nw, to_dev_dict(f)), nw.ContinuityOpts(**od))
    vals, rhs = ls.to_host()
    check_close(vals, ref["vals"], ref["vabs"], "values")
    check_close(rhs, ref["rhs"], ref["rabs"], "rhs")


@pytest.mark.parametrize("limiter,tanh,alpha", [(0, 0, 0.0), (1, 1, 0.0), (1, 0, 0.3), (0, 1, 0.3)])
@pytest.mark.parametrize("dims", [(1, 1, 1), (34, 34, 34), (36, 36, 36)])
def test_scalar(nw, orc, dims, limiter, tanh, alpha):
    mesh = nw.Mesh(*dims, jitter=0.04, seed=6)
    assert (mesh.num_edges > 131072) == (dims[0] == 36)
    rng = np.random.default_rng(8)
    N = mesh.num_nodes
    f = dict(coords=mesh.coords, velocity=rng.normal(size=(N, 3)), q=rng.uniform(size=N),
             dqdx=rng.normal(size=(N, 3)), density=rng.uniform(0.5, 2, N), diff=rng.uniform(1e-3, 1e-1, N),
             area=mesh.area, mdot=rng.normal(size=mesh.num_edges))
    od = dict(alpha=alpha, alpha_upw=0.7, upw_factor=1.0, relax=0.8, hybrid_factor=1.0, use_limiter=limiter,
              tanh_form=tanh, tanh_trans=2.0, tanh_width=4.0)
    ref = oracle_scalar(orc, mesh.edges, mesh.nalu_id, f, od)
    ls = _linsys(nw, N, mesh.edges)
    ls.assemble_scalar(scalar_fields(nw, to_dev_dict(f)), nw.ScalarOpts(**od))
    vals, rhs = ls.to_host()
    check_close(vals, ref["vals"], ref["vabs"], "scalar values")
    check_close(rhs, ref["rhs"], ref["rabs"], "scalar rhs")
