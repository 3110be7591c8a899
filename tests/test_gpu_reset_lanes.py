"""Row resets with eight and with four lanes a row: few rows, many short ones and
many long ones, numbers of rows around the line and around a block."""
import numpy as np
import pytest

from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nd,tets,shape", [(1, False, (17, 17, 16)), (3, False, (12, 11, 9)), (3, True, (12, 11, 9))])
def test_reset_of_many_rows(nw, nd, tets, shape):
    mesh = nw.Mesh(*shape, tets=tets)
    ls = nw.LinearSystem(nd)
    ls.build_edge_graph(mesh.num_nodes, mesh.edges)
    ls.finalize()
    nr, nz = ls.sizes()
    assert nr > 4096 and (nz / nr >= 32) == tets
    rp, ci = ls.graph()
    rng = np.random.default_rng(3)
    row = np.repeat(np.arange(nr), np.diff(rp))
    for n in (4096 // nd, 4096 // nd + 1, mesh.num_nodes):
        v, b = rng.normal(size=nz), rng.normal(size=nr)
        ls.from_host(v, b)
        nodes = rng.permutation(mesh.num_nodes)[:n].astype(np.int64)
        ls.reset_rows(n, dev(nodes), 0, nd, 2.5, -0.5)
        vals, rhs = ls.to_host()
        hit = np.zeros(nr, bool)
        hit[(nodes[:, None] * nd + np.arange(nd)).ravel()] = True
        np.testing.assert_array_equal(vals, np.where(hit[row], np.where(ci == row, 2.5, 0.0), v))
        np.testing.assert_array_equal(rhs, np.where(hit, -0.5, b))
