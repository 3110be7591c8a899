"""The continuity rows for each non-orthogonal factor (the default 1 has its own
kernel) against the reference's formulas. Tolerance as in the parity tests."""
import numpy as np
import pytest

from gpu_util import check_close, continuity_fields, oracle_continuity, to_dev_dict

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("noc", [0.0, 0.4, 1.0])
@pytest.mark.parametrize("dims", [(1, 1, 1), (9, 8, 7)])
def test_continuity_rows(nw, orc, noc, dims):
    mesh = nw.Mesh(*dims, tets=True, jitter=0.04, seed=4)
    rng = np.random.default_rng(5)
    N = mesh.num_nodes
    f = dict(coords=mesh.coords, velocity=rng.normal(size=(N, 3)), dpdx=rng.normal(size=(N, 3)),
             density=rng.uniform(0.5, 2, N), pressure=rng.normal(size=N), udiag=rng.uniform(1, 3, N),
             area=mesh.area)
    od = dict(noc_fac=noc, tau_scale=0.5, interp_together=1.0, solve_incompressible=0.0)
    ref = oracle_continuity(orc, mesh.edges, mesh.nalu_id, f, od)
    ls = nw.LinearSystem(1)
    ls.build_edge_graph(N, mesh.edges)
    ls.finalize()
    ls.zero_system()
    ls.assemble_continuity(continuity_fields(nw, to_dev_dict(f)), nw.ContinuityOpts(**od))
    vals, rhs = ls.to_host()
    check_close(vals, ref["vals"], ref["vabs"], f"continuity values, noc {noc}")
    check_close(rhs, ref["rhs"], ref["rabs"], f"continuity rhs, noc {noc}")
