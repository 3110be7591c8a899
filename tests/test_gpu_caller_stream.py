"""A solve leaves the caller's stream to the caller: while one thread solves on
a handle's stream, another may query that stream and launch work on it. The
solver's graphs are recorded elsewhere, so the queries succeed, every launched
kernel runs once, and the solve gives the bits of an undisturbed one."""
import threading

import pytest

from test_gpu_solver import _poisson_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["PREC_FP64", "PREC_MIXED"])
@pytest.mark.parametrize("pc", ["PC_JACOBI", "PC_SGS"])
def test_another_thread_uses_the_stream_of_a_solve(nw, precision, pc):
    import torch
    ls, _ = _poisson_system(nw, (20, 17, 9))
    stream = torch.cuda.Stream()
    ls.set_stream(stream.cuda_stream)
    ls.set_solver_cfg(nw.solver_cfg(preconditioner=getattr(nw, pc), precision=getattr(nw, precision), kspace=20,
                                    inner_kspace=20, max_iterations=600, tolerance=1e-13))
    n = ls.sizes()[0]
    alone, beside = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    ls.solve(alone)
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    stop, errors, launched = threading.Event(), [], [0]

    def other():
        try:
            while not stop.is_set():
                stream.query()
                with torch.cuda.stream(stream):
                    count.add_(1)
                launched[0] += 1
        except Exception as e:  # noqa: BLE001
            errors.append(str(e))

    t = threading.Thread(target=other)
    t.start()
    try:
        for _ in range(5):
            ls.solve(beside)
    finally:
        stop.set()
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    assert launched[0] > 0 and int(count) == launched[0]
    assert torch.equal(alone, beside)
