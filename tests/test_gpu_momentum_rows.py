"""The momentum row kernel at the edges of its work split: numbers of node
rows around the ten of a warp and the sixty of a block, odd CSR positions,
rows too long for the staging area (hub nodes), repeated assembly into a
system that holds values, and the same through edge and row ranges. Against
the oracle, with the parity bounds of every assembly test."""
import numpy as np
import pytest

from gpu_util import check_close, momentum_fields, oracle_momentum, to_dev_dict

pytestmark = pytest.mark.gpu

OPTS = [dict(alpha=0.0, alpha_upw=1.0, upw_factor=1.0, relax=0.7, include_div_u=1.0, use_limiter=1),
        dict(alpha=0.3, alpha_upw=0.8, upw_factor=0.9, relax=1.0, include_div_u=0.0, use_limiter=0)]


def _graph(n, hubs, seed):
    """A ring of n nodes, a few chords, and `hubs` nodes joined to all others."""
    rng = np.random.default_rng(seed)
    e = {(i, (i + 1) % n) for i in range(n) if n > 1 and i != (i + 1) % n}
    e |= {(int(a), int(b)) for a, b in rng.integers(0, n, (n, 2)) if a != b}
    e |= {(h, i) for h in range(hubs) for i in range(n) if i != h}
    return np.array(sorted({(min(a, b), max(a, b)) for a, b in e}), np.int64)


@pytest.mark.parametrize("n,hubs", [(2, 0), (9, 0), (10, 0), (11, 0), (59, 0), (60, 0), (61, 1), (301, 0), (701, 3)])
@pytest.mark.parametrize("k", [0, 1])
def test_rows_match_oracle(nw, orc, n, hubs, k):
    edges = _graph(n, hubs, 7 * n + k)
    rng = np.random.default_rng(n)
    E = len(edges)
    x = rng.normal(size=(n, 3))
    dx = x[edges[:, 1]] - x[edges[:, 0]]
    f = dict(coords=x, velocity=rng.normal(size=(n, 3)), dudx=rng.normal(size=(n, 9)),
             viscosity=rng.uniform(1e-3, 1e-1, n), density=np.ones(n), mask=rng.choice([0.0, 1.0], n),
             area=dx + 0.1 * rng.normal(size=(E, 3)), mdot=rng.normal(size=E), pecfac=rng.uniform(size=E))
    ref = oracle_momentum(orc, edges, np.arange(1, n + 1), f, OPTS[k])
    ls = nw.LinearSystem(3)
    ls.build_edge_graph(n, edges)
    ls.finalize()
    mf, o = momentum_fields(nw, to_dev_dict(f)), nw.MomentumOpts(**OPTS[k])
    ls.zero_system()
    ls.assemble_momentum(mf, o)
    v, b = ls.to_host()
    check_close(v, ref["vals"], ref["vabs"], f"values n {n} hubs {hubs}")
    check_close(b, ref["rhs"], ref["rabs"], f"rhs n {n} hubs {hubs}")
    ls.assemble_momentum(mf, o)  # adds
    v2, b2 = ls.to_host()
    np.testing.assert_array_equal(v2, v + v)
    np.testing.assert_array_equal(b2, b + b)
    # edge ranges and row ranges give the same bits
    ls.zero_system()
    for e0 in range(0, E, 97):
        ls.assemble_momentum_range(mf, o, e0, min(E, e0 + 97))
    for r0 in range(0, n, 13):
        ls.assemble_momentum_rows_range(o, r0, min(n, r0 + 13))
    v3, b3 = ls.to_host()
    np.testing.assert_array_equal(v3, v)
    np.testing.assert_array_equal(b3, b)
