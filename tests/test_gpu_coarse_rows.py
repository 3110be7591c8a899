"""The network's coarse-graph kernels at sizes where their launch shapes end:
one coarse row, fewer than a block, several blocks, and enough blocks that the
final sums take their block-wide tree (more than 32 partial sums of 256 rows);
rows shorter and longer than one batch of gathers. Forward output and loss
against the oracle with the same BF16 rounding points, tolerances as in
test_gpu_learned."""
import numpy as np
import pytest

from gpu_util import dev
from oracle import learned_oracle as lo
from test_gpu_learned import _poisson, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,passes,least", [((2, 2, 2), 2, 1), ((9, 8, 7), 1, 5), ((22, 21, 20), 1, 257),
                                                ((53, 52, 51), 1, 8193)])
def test_forward_and_loss(nw, shape, passes, least):
    import torch
    ls = _poisson(nw, shape)
    net = nw.Learned(seed=5)
    net.configure(agg_passes=passes)
    ls.attach_learned(net)
    cg = ls.coarse_graph()
    nc = cg["nc"]
    assert nc >= least
    rng = np.random.default_rng(12)
    H = lo.H
    net.set_params(np.concatenate([rng.uniform(-1.7, 1.7, 2 * H), rng.uniform(-0.2, 0.2, 6 * H * H),
                                   rng.uniform(-0.2, 0.2, H)]).astype(np.float32))
    rc = rng.normal(size=nc).astype(np.float32)
    ea, ca = 40.0, 25.0
    rc_d = dev(rc)
    ec_d = torch.zeros(nc, dtype=torch.float32, device="cuda")
    net.forward(ls, rc_d, ec_d)
    L, _ = net.loss_grad(ls, rc_d, ea, ca)
    Lb, _, ecb = lo.loss_and_grad(net.params().astype(np.float64), cg, rc, ea, ca, bf16_points=True)
    assert _rel(ec_d.cpu().numpy().astype(np.float64), ecb) <= 5e-3
    Ac = lo.coarse_operator(cg)
    lscale = (np.abs(ecb) @ np.abs(Ac) @ np.abs(ecb) + 2 * np.abs(ecb) @ np.abs(rc) + ca) / ea
    assert abs(L - Lb) <= 5e-3 * lscale
