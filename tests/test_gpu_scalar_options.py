"""Every specialisation of the scalar edge kernel (limiter, tanh Peclet
function, alpha zero or not) against the oracle, with mass flows of both signs
and zero, Peclet numbers from below 1e-3 to above 1e3 (both ends of the blending
functions), a relaxation factor, and node counts around a row block of 128."""
import numpy as np
import pytest

from gpu_util import check_close, oracle_scalar, scalar_fields, to_dev_dict

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (7, 3, 3), (42, 2, 1), (13, 9, 8)])
@pytest.mark.parametrize("k", range(8))
def test_scalar_specialisations_match_oracle(nw, orc, shape, k):
    mesh = nw.Mesh(*shape, jitter=0.05, seed=3)
    rng = np.random.default_rng(17 * k + mesh.num_nodes)
    N, E = mesh.num_nodes, mesh.num_edges
    f = dict(coords=mesh.coords, velocity=rng.normal(size=(N, 3)), q=rng.uniform(size=N), dqdx=rng.normal(size=(N, 3)),
             density=rng.uniform(0.8, 1.2, N), diff=10.0 ** rng.uniform(-5, 3, N), area=mesh.area,
             mdot=rng.normal(size=E) * rng.choice([0.0, 1.0], E, p=[0.2, 0.8]))
    od = dict(alpha=0.3 if k & 1 else 0.0, alpha_upw=0.7, upw_factor=0.9, relax=0.6, hybrid_factor=1.0,
              use_limiter=(k >> 2) & 1, tanh_form=(k >> 1) & 1, tanh_trans=2.0, tanh_width=4.0)
    ref = oracle_scalar(orc, mesh.edges, np.arange(1, N + 1), f, od)
    ls = nw.LinearSystem(1)
    ls.build_edge_graph(N, mesh.edges)
    ls.finalize()
    ls.zero_system()
    ls.assemble_scalar(scalar_fields(nw, to_dev_dict(f)), nw.ScalarOpts(**od))
    v, b = ls.to_host()
    check_close(v, ref["vals"], ref["vabs"], f"scalar values {od}", rel_floor=2.0)
    check_close(b, ref["rhs"], ref["rabs"], f"scalar rhs {od}", rel_floor=2.0)
