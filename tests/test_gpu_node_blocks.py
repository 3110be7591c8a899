"""Node kernels on both sides of the 16,384 nodes up to which they run in small
blocks: time terms, diagonal and its projection factor on a chain of nodes,
against the formulas in NumPy FP64 (1e-14 of the summed magnitudes: four
products and a division each)."""
import numpy as np
import pytest

from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65, 16384, 16385])
@pytest.mark.parametrize("kind", ["scalar", "continuity", "momentum"])
def test_time_terms(nw, kind, n):
    nd = 3 if kind == "momentum" else 1
    rng = np.random.default_rng(n)
    ls = nw.LinearSystem(nd)
    ls.build_edge_graph(n, np.stack([np.arange(n - 1), np.arange(1, n)], 1))
    ls.finalize()
    rho, vol = rng.uniform(0.5, 1.5, (3, n)), rng.uniform(0.5, 1.5, (3, n))
    q, dpdx = rng.normal(size=(3, n, nd)), rng.normal(size=(n, 3))
    dt, g = 0.05, (1.5, -2.0, 0.5)
    ls.zero_system()
    ls.assemble_mass_bdf(kind, [dev(a) for a in rho], [dev(a) for a in vol],
                         q=None if kind == "continuity" else [dev(a if nd == 3 else a[:, 0]) for a in q],
                         dpdx=dev(dpdx) if nd == 3 else None, dt=dt, gamma=g)
    m = [gk * rho[t] * vol[t] / dt for gk, t in zip(g, (2, 1, 0))]
    if kind == "continuity":
        terms = [-mk[:, None] * g[0] / dt for mk in m]
    else:
        terms = [-mk[:, None] * q[t] for mk, t in zip(m, (2, 1, 0))]
        if nd == 3:
            terms.append(-dpdx * vol[2][:, None])
    v, b = ls.to_host()
    err = np.abs(b.reshape(n, nd) - sum(terms))
    assert np.all(err <= 1e-14 * sum(np.abs(t) for t in terms))
    import torch
    d = torch.zeros(n, dtype=torch.float64, device="cuda")
    ls.extract_diagonal(d, dof=nd - 1)
    lhs = np.zeros(n) if kind == "continuity" else m[0]
    np.testing.assert_allclose(d.cpu().numpy(), lhs, rtol=1e-14)
    u0 = rng.uniform(1.0, 2.0, n)
    u = dev(u0)
    ls.udiag_postprocess(dev(rho[2]), dev(vol[2]), u, dt, g[0], 0.7)
    pts = g[0] / dt
    quotient = u0 / (rho[2] * vol[2])
    np.testing.assert_allclose(u.cpu().numpy(), (quotient - pts) * 0.7 + pts, rtol=0, atol=1e-14 * (pts + quotient).max())
