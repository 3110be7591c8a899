"""GMRES cycles against the solver's launch chunks (two iterations a graph):
restart lengths and iteration limits that end inside, at and beside a chunk,
several cycles a solve, against the oracle's solver in the GPU's operation
order (iteration count, history and solution to 1e-12)."""
import pytest

from test_gpu_solver import _check_gpu_order, _gpu_order, _poisson_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kspace,iters", [(1, 5), (2, 7), (3, 11), (4, 4), (5, 24), (20, 1), (20, 2), (20, 41)])
def test_cycles_end_anywhere_in_a_chunk(nw, orc, kspace, iters):
    import torch
    ls, _ = _poisson_system(nw, (7, 7, 3))
    ls.set_solver_cfg(nw.solver_cfg(preconditioner=1, kspace=kspace, max_iterations=iters, tolerance=1e-11))
    x = torch.zeros(ls.sizes()[0], dtype=torch.float64, device="cuda")
    for _ in range(2):  # the second solve updates the first one's graph
        rep = ls.solve(x)
        _check_gpu_order(rep, ls.residual_history(), x.cpu().numpy(), _gpu_order(orc, ls, 0, 1, kspace, iters, 1e-11),
                         f"kspace {kspace}, {iters} iterations")
