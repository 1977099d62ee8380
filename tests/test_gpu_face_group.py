"""Simpson face fluxes, eight polygons to a warp, against the CPU oracle bit
for bit: every face kind (axis-aligned, tilted, triangles, warped, refined),
planes that move across a face, along it and not at all, one to many faces."""

import numpy as np
import pytest

from geometricvofext_gb300 import capi, harness as H, meshgen as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n", [("hex", 5), ("hex", 12), ("jitter", 5), ("jitter", 9), ("tet", 5), ("checker", 6),
                                    ("refined", 8)])
def test_face_fluxes_bitexact(kind, n):
    m = mg.make_mesh(kind, n)
    rng = np.random.default_rng(11)
    g = capi.Simplic(m, n_alpha_bounds=0, clip=0, record_cut_faces=1)
    o = O.Oracle(m, n_alpha_bounds=0, clip=False)
    x = m.C
    fields = (rng.random(m.n_cells), np.clip(0.5 - (x[:, 2] - 0.43) * 3, 0, 1),
              np.clip(0.5 - (x.sum(1) - 1.3) * 2, 0, 1), np.where(np.arange(m.n_cells) == m.n_cells // 2, 0.4, 0.0))
    flows = (H.DeformationFlow(m), H.TranslationFlow(m, U=(0.5, 0.5, 0.5)), H.TranslationFlow(m, U=(1.0, 0.0, 0.0)),
             H.TranslationFlow(m, U=(0.0, 0.0, -1.0)))
    for flow in flows:
        dt = H.cfl_delta_t(m, flow.phi0)
        for a0 in fields:
            for scale in (1.0, 1e-9):  # across faces within the step, and hardly moving
                phi, U = flow.phi0 * scale, flow.U0 * scale
                g.reconstruct(a0)
                o.reconstruct(a0)
                ag = g.advect(a0, phi, U, dt, U_boundary=flow.Ub * scale)
                ao = o.advect(a0, phi, U, dt, U_boundary=flow.Ub * scale)
                np.testing.assert_array_equal(g.alpha_phi(), o.alpha_phi())
                np.testing.assert_array_equal(ag, ao)
                np.testing.assert_array_equal(g.cut_faces(), o.cut_faces())
