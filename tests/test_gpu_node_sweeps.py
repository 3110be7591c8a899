"""Multicolour symmetric Gauss-Seidel on systems with three rows a node, where
one kernel relaxes a node's rows in turn: the preconditioner and whole GMRES
solves against the oracle in the GPU's operation order (which relaxes class by
class), on two colours (hexes), several (tets), one node, and nodes that are
not a multiple of a block or slice."""
import numpy as np
import pytest

from test_gpu_solver import _check_gpu_order, _gpu_order

pytestmark = pytest.mark.gpu


def _system(nw, shape, tets, renumber):
    import torch
    mesh = nw.Mesh(*shape, tets=tets, jitter=0.05, seed=4, renumber=renumber, renumber_seed=2)
    ls = nw.LinearSystem(3)
    ls.build_edge_graph(mesh.num_nodes, mesh.edges)
    ls.finalize()
    rp, ci = ls.graph()
    rng = np.random.default_rng(8)
    v = rng.uniform(-1.0, 1.0, len(ci))
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    v[rows == ci] = 1.0 + np.bincount(rows, np.abs(v), len(rp) - 1) * rng.uniform(0.6, 0.9, len(rp) - 1)
    ls.from_host(values=v, rhs=rng.normal(size=len(rp) - 1))
    return ls, rp, ci, v


@pytest.mark.parametrize("shape,tets,renumber", [((1, 1, 1), False, 0), ((3, 2, 2), False, 0), ((9, 8, 7), False, 0),
                                                 ((5, 4, 3), True, 0), ((8, 7, 6), True, 1)])
def test_three_rows_a_node(nw, orc, shape, tets, renumber):
    import torch
    ls, rp, ci, v = _system(nw, shape, tets, renumber)
    n = len(rp) - 1
    # one application, row by row in the sweep's order
    order, nc = ls.sgs_order()
    cp = ls.sgs_classes()
    x = np.random.default_rng(1).normal(size=n)
    y = np.zeros(n)
    diag = v[np.flatnonzero(ci == np.repeat(np.arange(n), np.diff(rp)))]
    last = order[cp[nc - 1]:]
    for i in list(order) + list(order[::-1][len(last):]):
        s = slice(rp[i], rp[i + 1])
        y[i] = (x[i] - v[s] @ y[ci[s]] + diag[i] * y[i]) / diag[i]
    xd = torch.from_numpy(x).cuda()
    yd = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")  # nothing stale may be read
    ls.precond_apply(nw.PC_SGS, xd, yd)
    torch.cuda.synchronize()
    assert np.abs(yd.cpu().numpy() - y).max() <= 1e-13 * np.abs(y).max()
    # whole solves: FP64 to the bit pattern of the class order, mixed to the residual
    ls.set_solver_cfg(nw.solver_cfg(preconditioner=2, kspace=30, max_iterations=60, tolerance=1e-9))
    xs = torch.zeros(n, dtype=torch.float64, device="cuda")
    rep = ls.solve(xs)
    _check_gpu_order(rep, ls.residual_history(), xs.cpu().numpy(), _gpu_order(orc, ls, 0, 2, 30, 60, 1e-9, lanes=32),
                     f"{shape} tets {tets}")
    for prec in (nw.PREC_MIXED, nw.PREC_MIXED_BF16):
        ls.set_solver_cfg(nw.solver_cfg(preconditioner=2, precision=prec, kspace=30, max_iterations=200,
                                        tolerance=1e-10))
        rep = ls.solve(xs)
        _, b = ls.to_host()
        r = b - np.add.reduceat(v * xs.cpu().numpy()[ci], rp[:-1])
        assert rep.converged == 1 and np.linalg.norm(r) <= 1.01e-10 * np.linalg.norm(b)
