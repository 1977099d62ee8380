"""A block whose interior is a lattice but whose boundary cells are joined by a
further face (bottom to top of one column, numbered after the others) is not
taken for one, and its update is the oracle's, bit for bit."""

import numpy as np
import pytest

from geometricvofext_gb300 import capi, harness as H, meshgen as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _joined(n, i, j):
    """hex_mesh(n) with the bottom face of column (i, j) made the face between
    its lowest and its highest cell, and the top face left out."""
    m = mg.hex_mesh(n)
    nfi = m.n_internal_faces
    low, high = i + n * j, i + n * (j + n * (n - 1))
    bot = next(f for f in range(nfi, m.n_faces) if m.owner[f] == low and m.Cf[f, 2] < 1e-9)
    top = next(f for f in range(nfi, m.n_faces) if m.owner[f] == high and m.Cf[f, 2] > 1 - 1e-9)
    order = np.r_[np.arange(nfi), bot, [f for f in range(nfi, m.n_faces) if f not in (bot, top)]]
    d = mg.PolyMesh(points=m.points, face_offsets=np.arange(order.size + 1, dtype=np.int32) * 4,
                    face_points=m.faces_dense()[order].astype(np.int32).ravel(), owner=m.owner[order].astype(np.int32),
                    neighbour=np.r_[m.neighbour, high].astype(np.int32), n_cells=m.n_cells, patches=[], kind="hex")
    d.C, d.V, d.h = m.C, m.V, m.h
    d.Cf, d.Sf, d.magSf = m.Cf[order], m.Sf[order], m.magSf[order]
    return d


@pytest.mark.parametrize("n,i,j", [(5, 2, 2), (9, 1, 6), (12, 5, 3)])
def test_update_of_a_block_joined_at_its_boundary(n, i, j):
    m = _joined(n, i, j)
    rng = np.random.default_rng(n)
    phi = rng.standard_normal(m.n_faces) * m.magSf
    dt = 0.1 * m.h
    U, Ub = np.zeros((m.n_cells, 3)), np.zeros((m.n_boundary_faces, 3))
    g, o = capi.Simplic(m, n_alpha_bounds=3, clip=0), O.Oracle(m, n_alpha_bounds=3, clip=False)
    # (below the mixed range: the update alone)
    for a in (1e-9 * rng.random(m.n_cells), np.where(rng.random(m.n_cells) < 0.3, 1e-9, 0.0)):
        g.reconstruct(a)
        o.reconstruct(a)
        np.testing.assert_array_equal(g.advect(a, phi, U, dt, U_boundary=Ub), o.advect(a, phi, U, dt, U_boundary=Ub))
        np.testing.assert_array_equal(g.alpha_phi(), o.alpha_phi())
    assert g.mesh_info()[1] == 0
