"""Hex8 sub-control surfaces and volumes (closed forms of the trilinear map)
against the oracle's fans and Grandy volumes on strongly distorted hexes,
one element up to a few hundred, near and far from the origin.

Tolerance: both sides round products of differences of coordinates of size
c over cells of size h; the differences are exact to about eps c, so an area
is off by a few eps c h and a volume by a few eps c h^2."""
import numpy as np
import pytest

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("shape,jitter,opts", [((1, 1, 1), 0.0, {}), ((2, 1, 3), 0.3, {}), ((7, 6, 5), 0.3, {}),
                                               ((5, 4, 6), 0.2, dict(stretch_z=1.3, lx=100.0, ly=50.0, lz=20.0))])
def test_distorted_hexes_against_fans_and_grandy(nw, orc, shape, jitter, opts):
    mesh = nw.Mesh(*shape, jitter=jitter, seed=9, **opts)
    oedges, ee = orc.hex8_edges(mesh.conn, mesh.num_nodes)
    area, vol = orc.hex8_geometry(mesh.coords, mesh.conn, ee, oedges)
    key = {tuple(e): i for i, e in enumerate(oedges.tolist())}
    perm = np.array([key[tuple(e)] for e in mesh.edges.tolist()])
    c = np.abs(mesh.coords).max()
    h = np.linalg.norm(mesh.coords[mesh.edges[:, 1]] - mesh.coords[mesh.edges[:, 0]], axis=1).max()
    assert np.abs(mesh.area - area[perm]).max() <= 64 * EPS * c * h
    # Grandy's formula weighs its terms by whole coordinates
    assert np.abs(mesh.dualvol - vol).max() <= 256 * EPS * c * h * h
    ext = mesh.coords.max(0) - mesh.coords.min(0)
    assert abs(mesh.dualvol.sum() - ext.prod()) <= 1e-12 * ext.prod()
