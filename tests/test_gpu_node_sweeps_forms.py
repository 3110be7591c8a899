"""The node-wise Gauss-Seidel sweep with two and with three rows a node, on two
colours (a path; a star, whose hub's rows are longer than many batches) and on
many colours with rows longer than a batch (a clique joined to a path): one
application against the sweep row by row in class order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRAPHS = {"star": (70, [(0, k) for k in range(1, 70)]), "path": (131, [(k, k + 1) for k in range(130)]),
          "clique": (90, [(a, b) for a in range(14) for b in range(a + 1, 14)] + [(k, k + 1) for k in range(13, 89)])}


@pytest.mark.parametrize("nd", [2, 3])
@pytest.mark.parametrize("graph", sorted(GRAPHS))
def test_one_application(nw, nd, graph):
    import torch
    N, edges = GRAPHS[graph]
    ls = nw.LinearSystem(nd)
    ls.build_edge_graph(N, np.array(edges, np.int64).reshape(-1, 2))
    ls.finalize()
    rp, ci = ls.graph()
    n = len(rp) - 1
    rng = np.random.default_rng(8)
    v = rng.uniform(-1.0, 1.0, len(ci))
    rows = np.repeat(np.arange(n), np.diff(rp))
    v[rows == ci] = 1.0 + np.bincount(rows, np.abs(v), n) * rng.uniform(0.6, 0.9, n)
    diag = v[rows == ci]
    ls.from_host(values=v, rhs=np.zeros(n))
    order, nc = ls.sgs_order()
    last = order[ls.sgs_classes()[nc - 1]:]
    x, y = rng.normal(size=n), np.zeros(n)
    for i in list(order) + list(order[::-1][len(last):]):
        s = slice(rp[i], rp[i + 1])
        y[i] = (x[i] - v[s] @ y[ci[s]] + diag[i] * y[i]) / diag[i]
    out = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")  # nothing stale may be read
    ls.precond_apply(nw.PC_SGS, torch.from_numpy(x).cuda(), out)
    torch.cuda.synchronize()
    assert np.abs(out.cpu().numpy() - y).max() <= 1e-13 * np.abs(y).max()
