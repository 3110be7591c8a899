"""The learned cycle's kernels start under the one before them (sweeps,
residual, restriction, network layers with the TMA product, coarse operator,
prolongation). A process in which every launch waits for the kernel before it
(CUDA_LAUNCH_BLOCKING) gives the same bits: solves of one-iteration cycles
(plain launches throughout) and of longer ones (graphs after the first two
iterations), for both smoothers, the three coarse directions, FP32 and BF16
sweeps, each after the values have changed."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
HERE = Path(__file__).resolve().parent

SCRIPT = '''
import hashlib, sys
sys.path[:0] = [{root!r}, {here!r}]
import torch
import __graft_entry__ as g
nw = g._package()
from test_gpu_solver import _poisson_system
for smoother in (0, 1):
    for mode in (0, 1, 2):
        net = nw.Learned(seed=3)
        net.configure(smoother=smoother)
        net.set_coarse_direction(mode)
        ls, _ = _poisson_system(nw, (20, 17, 9))
        ls.attach_learned(net)
        v, b = ls.to_host()
        x = torch.zeros(ls.sizes()[0], dtype=torch.float64, device="cuda")
        k = 0
        for precision in (nw.PREC_MIXED, nw.PREC_MIXED_BF16):
            for kspace in (1, 12):
                k += 1
                ls.from_host(v * (1.0 + 0.25 * k), b)
                ls.set_solver_cfg(nw.solver_cfg(method=nw.FGMRES, preconditioner=nw.PC_LEARNED, precision=precision,
                                                kspace=kspace, inner_kspace=kspace, max_iterations=24,
                                                tolerance=1e-14))
                rep = ls.solve(x)
                # the history holds the learned cycles', also where the solve falls back
                hist = ls.residual_history()
                bits = hashlib.sha256(x.cpu().numpy().tobytes() + hist.tobytes()).hexdigest()
                print(smoother, mode, precision, kspace, rep.iterations, bool(torch.isfinite(x).all()), bits)
'''


def _lines(blocking):
    env = dict(os.environ)
    env.pop("CUDA_LAUNCH_BLOCKING", None)
    if blocking:
        env["CUDA_LAUNCH_BLOCKING"] = "1"
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=str(HERE.parent), here=str(HERE))], env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout.split("\n")[:-1]


def test_bits_do_not_depend_on_the_overlap():
    idle, overlapped = _lines(True), _lines(False)
    assert len(idle) == 24 and all(" True " in line for line in idle)
    assert idle == overlapped
