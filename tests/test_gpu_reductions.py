"""The solver's multi-dots and multi-axpys at the edges of their launch
shapes: rows below, at and above a block of 256, and on both sides of the
sizes where the multi-axpy changes its elements per thread (4 x 152 and 24 x
152 blocks of 256 rows); restart length 20, so that every tile width of the
multi-dot (1 to 8 vectors) occurs. Against the oracle's solver in the GPU's
operation order (iteration count, history and solution to 1e-12), and the
mixed-precision solver's FP64 residual."""
import numpy as np
import pytest

from test_gpu_solver import _check_gpu_order, _gpu_order, _poisson_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,iters", [((2, 1, 1), 8), ((7, 7, 3), 45), ((16, 16, 2), 45), ((40, 31, 23), 45),
                                         ((63, 63, 36), 24), ((63, 63, 37), 24), ((127, 127, 55), 21),
                                         ((127, 127, 56), 21)])
def test_gmres_reductions_match_oracle_order(nw, orc, shape, iters):
    import torch
    ls, _ = _poisson_system(nw, shape)
    ls.set_solver_cfg(nw.solver_cfg(preconditioner=1, kspace=20, max_iterations=iters, tolerance=1e-11))
    x = torch.zeros(ls.sizes()[0], dtype=torch.float64, device="cuda")
    rep = ls.solve(x)
    _check_gpu_order(rep, ls.residual_history(), x.cpu().numpy(), _gpu_order(orc, ls, 0, 1, 20, iters, 1e-11),
                     f"{shape}")


@pytest.mark.parametrize("shape", [(2, 1, 1), (7, 7, 3), (40, 31, 23)])
def test_mixed_reductions_reach_the_fp64_residual(nw, shape):
    import torch
    ls, _ = _poisson_system(nw, shape)
    ls.set_solver_cfg(nw.solver_cfg(preconditioner=2, precision=nw.PREC_MIXED, kspace=50, max_iterations=4000,
                                    tolerance=1e-9))
    x = torch.zeros(ls.sizes()[0], dtype=torch.float64, device="cuda")
    rep = ls.solve(x)
    assert rep.converged == 1
    rp, ci = ls.graph()
    v, b = ls.to_host()
    xh = x.cpu().numpy()
    r = b - np.add.reduceat(v * xh[ci], rp[:-1])
    assert np.linalg.norm(r) <= 1.01e-9 * np.linalg.norm(b)
