"""Kernels that share a row between lanes, at rows that do not fill or overfill
them: the open continuity boundary with 1 to more than 12 face points a row
(against the oracle) and the reset of rows over every range of unknowns."""
import numpy as np
import pytest

from gpu_util import check_close, dev
from test_gpu_boundary import _mesh, _node_fields, _oracle_sum, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("repeat", [1, 2, 3])
@pytest.mark.parametrize("kind", ["hex", "tets"])
def test_open_rows_of_many_points(nw, orc, kind, repeat):
    mesh = _mesh(nw, kind)
    rng = np.random.default_rng(21)
    f = _node_fields(mesh, rng)
    ipn, area = mesh.face_ips(("x+", "y-", "z+"))
    ipn = np.concatenate([ipn] * repeat)
    area = np.concatenate([area * (1.0 + 0.3 * k) for k in range(repeat)])
    dynp = rng.normal(0, 0.1, len(ipn))
    ls = _system(nw, mesh, 1)
    ss = ls.sideset(ipn)
    d = {k: dev(v) for k, v in dict(f, area=area, dynp=dynp).items()}
    fld = nw.ContinuityOpenFields(*(d[k].data_ptr() for k in ("coords", "velocity", "dpdx", "density", "pressure",
                                                               "pressure_bc", "udiag", "area", "dynp")))
    oo = dict(tau_scale=0.7, noc_fac=0.6, pstab_fac=1.0, mdot_corr=0.01, solve_incompressible=0.0)
    ls.assemble_continuity_open(ss, fld, nw.ContinuityOpenOpts(**oo))
    vals, rhs = ls.to_host()
    args = (ipn, f["coords"], f["velocity"], f["dpdx"], f["density"], f["pressure"], f["pressure_bc"],
            f["udiag"], area, dynp, orc.ContinuityOpenOpts(**oo))
    ref = _oracle_sum(orc, mesh, 1, ipn, *orc.continuity_open_local(*args),
                      *orc.continuity_open_local(*args, mag=True))
    check_close(vals, ref[0], ref[2], "values")
    check_close(rhs, ref[1], ref[3], "rhs")


@pytest.mark.parametrize("nd,begin,end", [(1, 0, 1), (1, 0, 0), (3, 0, 3), (3, 1, 2), (3, 1, 3), (3, 2, 2)])
@pytest.mark.parametrize("n", [1, 17])
def test_reset_rows(nw, nd, begin, end, n):
    mesh = _mesh(nw, "tets")
    ls = _system(nw, mesh, nd)
    nr, nz = ls.sizes()
    rng = np.random.default_rng(22)
    v, b = rng.normal(size=nz), rng.normal(size=nr)
    ls.from_host(v, b)
    rp, ci = ls.graph()
    nodes = rng.permutation(mesh.num_nodes)[:n].astype(np.int64)
    ls.reset_rows(n, dev(nodes), begin, end, 2.5, -0.5)
    vals, rhs = ls.to_host()
    for r in (nd * k + d for k in nodes for d in range(begin, end)):  # serial mesh: row = node x unknowns + unknown
        v[rp[r]:rp[r + 1]] = np.where(ci[rp[r]:rp[r + 1]] == r, 2.5, 0.0)
        b[r] = -0.5
    np.testing.assert_array_equal(vals, v)
    np.testing.assert_array_equal(rhs, b)
    with pytest.raises(nw.NwError):
        ls.reset_rows(1, dev(np.array([mesh.num_nodes], np.int64)), begin, end, 1.0, 0.0)
