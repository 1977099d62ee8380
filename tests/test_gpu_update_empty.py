"""The tiled update of a lattice against the general one, bit for bit, where
empty neighbourhoods meet cells at work and the flux between them is not the
zero of the upwind formula: the upwind cell was cut when the interface was
found and emptied before the advect, or phi is not finite.  The general update
is taken on the same block with one detached cell appended."""

import numpy as np
import pytest

from geometricvofext_gb300 import capi, harness as H, meshgen as mg

pytestmark = pytest.mark.gpu


def _with_detached_cell(m):
    """m and one unit cube far from it: every face and cell of m keeps its number."""
    one = mg.hex_mesh(1)
    d = mg.PolyMesh(points=np.concatenate([m.points, one.points + 5.0]),
                    face_offsets=np.concatenate([m.face_offsets, m.face_offsets[-1] + one.face_offsets[1:]]).astype(np.int32),
                    face_points=np.concatenate([m.face_points, one.face_points + m.n_points]).astype(np.int32),
                    owner=np.concatenate([m.owner, one.owner + m.n_cells]).astype(np.int32), neighbour=m.neighbour,
                    n_cells=m.n_cells + 1, patches=m.patches, kind="hex")
    for k, off in (("C", 5.0), ("V", 0.0), ("Cf", 5.0), ("Sf", 0.0), ("magSf", 0.0)):
        setattr(d, k, np.concatenate([getattr(m, k), getattr(one, k) + off]))
    d.h = m.h
    return d


@pytest.mark.parametrize("n", [5, 9, 17])
@pytest.mark.parametrize("phi_values", ["finite", "non-finite"])
def test_fluxes_beside_empty_neighbourhoods(n, phi_values):
    m = mg.make_mesh("hex", n)
    d = _with_detached_cell(m)
    flow = H.DeformationFlow(m)
    dt = H.cfl_delta_t(m, flow.phi0)
    rng = np.random.default_rng(n)
    phi = flow.phi0 + 1e-3 * np.abs(flow.phi0).max() * rng.standard_normal(m.n_faces)
    pad = lambda a, k: np.concatenate([a, np.zeros((k,) + a.shape[1:])])  # noqa: E731
    t, g = capi.Simplic(m, n_alpha_bounds=3, clip=0), capi.Simplic(d, n_alpha_bounds=3, clip=0)
    assert t.mesh_info()[1] == n and g.mesh_info()[1] == 0  # a lattice, and none
    for _ in range(3):
        drops = rng.random(m.n_cells) < 0.06  # cut, then emptied
        a0 = np.where(rng.random(m.n_cells) < 0.03, rng.random(m.n_cells), 0.0)
        found, handed = np.where(drops, rng.uniform(0.1, 0.9, m.n_cells), a0), np.where(drops, 0.0, a0)
        ph = phi.copy()
        if phi_values == "non-finite":
            at = rng.random(m.n_faces) < 0.02
            ph[at] = rng.choice([np.inf, -np.inf], at.sum())
            # (a NaN is downwind of no cell, so no cut cell's flux through its face is ever formed)
            cut = found > 0.0
            beside = cut[m.owner]
            beside[: m.n_internal_faces] |= cut[m.neighbour]
            ph[(rng.random(m.n_faces) < 0.02) & ~beside] = np.nan
        t.reconstruct(found)
        g.reconstruct(pad(found, 1))
        at = t.advect(handed, ph, flow.U0, dt, U_boundary=flow.Ub)
        ag = g.advect(pad(handed, 1), pad(ph, 6), pad(flow.U0, 1), dt, U_boundary=pad(flow.Ub, 6))
        np.testing.assert_array_equal(at, ag[:-1])
        np.testing.assert_array_equal(t.alpha_phi(), g.alpha_phi()[:-6])
