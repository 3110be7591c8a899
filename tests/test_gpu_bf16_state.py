"""BF16 sweeps belong to the solve that asks for them: an FP64 solve with the
learned preconditioner, which sweeps in FP32, gives the bits of a fresh handle
after a NW_PREC_MIXED_BF16 solve; and the BF16 values kept between two such
solves follow the matrix."""
import numpy as np
import pytest

from test_gpu_solver import _poisson_system

pytestmark = pytest.mark.gpu


def _system(nw, net=None):
    ls, _ = _poisson_system(nw, (20, 17, 9))
    if net is not None:
        ls.attach_learned(net)
    return ls


def _cfg(nw, precision, pc):
    return nw.solver_cfg(method=nw.FGMRES, preconditioner=pc, precision=precision, kspace=20, inner_kspace=20,
                         max_iterations=400, tolerance=1e-8)


def _solve(nw, ls, precision, pc):
    import torch
    ls.set_solver_cfg(_cfg(nw, precision, pc))
    x = torch.zeros(ls.sizes()[0], dtype=torch.float64, device="cuda")
    rep = ls.solve(x)
    assert rep.converged == 1 and rep.fallback == 0
    return rep.iterations, x


@pytest.mark.parametrize("smoother", [0, 1])
def test_fp64_learned_solve_after_a_bf16_solve(nw, smoother):
    import torch
    net = nw.Learned(seed=3)
    net.configure(smoother=smoother)
    fresh = _solve(nw, _system(nw, net), nw.PREC_FP64, nw.PC_LEARNED)
    ls = _system(nw, net)
    _solve(nw, ls, nw.PREC_MIXED_BF16, nw.PC_LEARNED)
    used = _solve(nw, ls, nw.PREC_FP64, nw.PC_LEARNED)
    assert fresh[0] == used[0] and torch.equal(fresh[1], used[1])


@pytest.mark.parametrize("pc", ["PC_SGS", "PC_LEARNED"])
def test_bf16_values_follow_the_matrix(nw, pc):
    import torch
    kind = getattr(nw, pc)
    make = lambda: _system(nw, nw.Learned(seed=3) if pc == "PC_LEARNED" else None)  # noqa: E731
    ls = make()
    v, b = ls.to_host()
    other = v * np.random.default_rng(5).uniform(0.9, 1.1, v.size)
    rp, ci = ls.graph()
    diag = ci == np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    other[diag] *= 1.2
    first = _solve(nw, ls, nw.PREC_MIXED_BF16, kind)
    ls.from_host(other, b)
    second = _solve(nw, ls, nw.PREC_MIXED_BF16, kind)
    fresh = make()
    fresh.from_host(other, b)
    alone = _solve(nw, fresh, nw.PREC_MIXED_BF16, kind)
    assert second[0] == alone[0] and torch.equal(second[1], alone[1])
    assert not torch.equal(first[1], second[1])
