"""The tiled update of lattice meshes against the CPU oracle, bit for bit:
sizes below, at and past the tile edges, fields from exactly empty to spread
over the mesh, boundary values and sources."""

import numpy as np
import pytest

from geometricvofext_gb300 import capi, harness as H, meshgen as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 4, 5, 8, 9, 13, 16, 17])
@pytest.mark.parametrize("extra", ["none", "boundary", "sources"])
def test_update_bitexact_at_tile_edges(n, extra):
    m = mg.make_mesh("hex", n)
    flow = H.DeformationFlow(m)
    dt = H.cfl_delta_t(m, flow.phi0)
    rng = np.random.default_rng(n)
    kw = {}
    if extra == "boundary":
        kw = dict(alpha_boundary=rng.random(m.n_boundary_faces))
    if extra == "sources":
        kw = dict(Sp=-0.1 * rng.random(m.n_cells), Su=0.1 * rng.random(m.n_cells))
    # walls let some through, so boundary faces carry flux
    phi = flow.phi0 + 1e-3 * np.abs(flow.phi0).max() * rng.standard_normal(m.n_faces)
    sphere = H.sphere_alpha(m, (0.35, 0.35, 0.35), 0.2)
    for a0 in (sphere, rng.random(m.n_cells), rng.random(m.n_cells) * 10.0 ** rng.uniform(-320, 0, m.n_cells),
               np.where(rng.random(m.n_cells) < 0.5, 1.0, 0.0)):
        g, o = capi.Simplic(m, n_alpha_bounds=3, clip=0), O.Oracle(m, n_alpha_bounds=3, clip=False)
        ag, ao = a0.copy(), a0.copy()
        for _ in range(4):
            g.reconstruct(ag)
            o.reconstruct(ao)
            ag = g.advect(ag, phi, flow.U0, dt, U_boundary=flow.Ub, **kw)
            ao = o.advect(ao, phi, flow.U0, dt, U_boundary=flow.Ub, **kw)
            np.testing.assert_array_equal(ag, ao)
            np.testing.assert_array_equal(g.alpha_phi(), o.alpha_phi())
