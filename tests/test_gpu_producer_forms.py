"""The input producers' forms: the mass flow for each pair of non-orthogonal
and interpolation factors (the default pair has its own kernel) and the nodal
gradients on rows of one to many edges, against the formulas in NumPy FP64.
Tolerance 1e-12 of the summed magnitudes, as for every kernel in float pairs."""
import numpy as np
import pytest

from gpu_util import dev

pytestmark = pytest.mark.gpu


def _graph(n, seed):
    """Node k of a chain also joined to k mod 9 earlier nodes: rows of 1 to
    about 20 edges."""
    rng = np.random.default_rng(seed)
    e = {(k - 1, k) for k in range(1, n)}
    for k in range(2, n):
        e |= {(int(a), k) for a in rng.integers(0, k, k % 9)}
    return np.array(sorted(e), np.int64)


def _system(nw, n, seed):
    edges = _graph(n, seed)
    ls = nw.LinearSystem(1)
    ls.build_edge_graph(n, edges)
    ls.finalize()
    return ls, edges, np.random.default_rng(seed + 1)


@pytest.mark.parametrize("noc,interp", [(1.0, 1.0), (0.0, 1.0), (1.0, 0.0), (0.4, 0.3)])
@pytest.mark.parametrize("n", [2, 257])
def test_mass_flow_forms(nw, noc, interp, n):
    import torch
    ls, edges, rng = _system(nw, n, 5)
    E = len(edges)
    L, R = edges.T
    x, u, G = (rng.normal(size=(n, 3)) for _ in range(3))
    rho, ud, p = rng.uniform(0.8, 1.2, n), rng.uniform(0.5, 2.0, n), rng.normal(size=n)
    dx = x[R] - x[L]
    A = dx + 0.1 * rng.normal(size=(E, 3))
    iu = 1.0 / ud
    w = (A * A).sum(1) / (A * dx).sum(1)
    rip = 0.5 * (rho[L] + rho[R])
    ru = interp * 0.5 * (rho[R, None] * u[R] + rho[L, None] * u[L]) + (1 - interp) * rip[:, None] * 0.5 * (u[L] + u[R])
    g = 0.5 * (G[R] * iu[R, None] + G[L] * iu[L, None])
    pts = 0.5 * (iu[L] + iu[R])
    ref = -pts * (p[R] - p[L]) * w + ((ru + g) * A - noc * (A - w[:, None] * dx) * g).sum(1)
    mag = (np.abs(pts * w) * (np.abs(p[R]) + np.abs(p[L]))
           + ((np.abs(ru) + 2 * np.abs(g)) * np.abs(A) + np.abs(w[:, None] * dx * g)).sum(1))
    keep = [dev(a) for a in (x, u, G, rho, p, ud, A)]
    f = nw.ContinuityFields(*(t.data_ptr() for t in keep))
    out = torch.zeros(E, dtype=torch.float64, device="cuda")
    ls.compute_mdot(f, out, noc, interp)
    torch.cuda.synchronize()
    assert np.all(np.abs(out.cpu().numpy() - ref) <= 1e-12 * mag)


@pytest.mark.parametrize("dim1", [1, 3])
@pytest.mark.parametrize("n", [2, 131, 300])
@pytest.mark.parametrize("boundary", [False, True])
def test_gradients(nw, dim1, n, boundary):
    import torch
    ls, edges, rng = _system(nw, n, 9)
    E = len(edges)
    L, R = edges.T
    phi, A = rng.normal(size=(n, dim1)), rng.normal(size=(E, 3))
    A[rng.random((E, 3)) < 0.2] = 0.0
    V, B = rng.uniform(0.5, 2.0, n), rng.normal(size=(n, 3))
    ref, mag = np.zeros((n, dim1, 3)), np.zeros((n, dim1, 3))
    t = 0.5 * (phi[L] + phi[R])[:, :, None] * A[:, None]
    s = 0.5 * (np.abs(phi[L]) + np.abs(phi[R]))[:, :, None] * np.abs(A)[:, None]
    np.add.at(ref, L, t)
    np.add.at(ref, R, -t)
    np.add.at(mag, L, s)
    np.add.at(mag, R, s)
    if boundary:
        ref += phi[:, :, None] * B[:, None]
        mag += np.abs(phi[:, :, None] * B[:, None])
    out = torch.zeros((n, 3 * dim1), dtype=torch.float64, device="cuda")
    keep = [dev(a) for a in (phi, A, V, B)]
    ls.nodal_gradient(*keep[:3], out, keep[3] if boundary else None, dim1=dim1)
    torch.cuda.synchronize()
    err = np.abs(out.cpu().numpy().reshape(n, dim1, 3) - ref / V[:, None, None])
    assert np.all(err <= 1e-12 * mag / V[:, None, None])
