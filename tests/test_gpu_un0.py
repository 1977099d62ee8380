"""The interface speeds (velocity interpolated to the interface centres) of the
plain form through the fluxes they give, against the CPU oracle bit for bit:
lists on both sides of the line between eight lanes and one thread per cell,
cells of warped faces whose interface centre no tetrahedron holds, boundary
cells, and places and sizes at which single precision settles nothing."""

import numpy as np
import pytest

from geometricvofext_gb300 import capi, harness as H, meshgen as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _compare(m, fields):
    g, o = capi.Simplic(m, n_alpha_bounds=0, clip=0), O.Oracle(m, n_alpha_bounds=0, clip=False)
    rng = np.random.default_rng(2)
    flow = H.DeformationFlow(m)
    U, Ub = rng.standard_normal(flow.U0.shape), rng.standard_normal(flow.Ub.shape)
    dt = H.cfl_delta_t(m, flow.phi0)
    for a0 in fields:
        for ub in (Ub, None):
            g.reconstruct(a0)
            o.reconstruct(a0)
            ag = g.advect(a0, flow.phi0, U, dt, U_boundary=ub)
            ao = o.advect(a0, flow.phi0, U, dt, U_boundary=ub)
            np.testing.assert_array_equal(g.alpha_phi(), o.alpha_phi())
            np.testing.assert_array_equal(ag, ao)


@pytest.mark.parametrize("kind,n", [("hex", 28), ("jitter", 28), ("tet", 16), ("refined", 8), ("checker", 8)])
def test_both_sides_of_the_line(kind, n):
    import torch

    line = 96 * torch.cuda.get_device_properties(0).multi_processor_count
    m = mg.make_mesh(kind, n)
    rng = np.random.default_rng(7)
    a = rng.random(m.n_cells)
    fields = [a, np.where(np.arange(m.n_cells) == m.n_cells // 2, a, 0.0)]
    if m.n_cells > line:
        for k in (line, line + 1):
            b = np.zeros(m.n_cells)
            pick = rng.choice(m.n_cells, k, replace=False)
            b[pick] = rng.uniform(1e-3, 0.999, k)
            fields.append(b)
    _compare(m, fields)


@pytest.mark.parametrize("scale,offset", [((1, 0.01, 30), (-5, 0.3, 2)), ((1e-7, 1e-7, 1e-7), (0, 0, 0)),
                                          ((1, 1, 1), (3e7, 0, 0)), ((1e9, 1e9, 1e9), (0, 0, 0))])
def test_sizes_and_places(scale, offset):
    m = mg.hex_mesh(6, metrics=False)
    m.points = m.points * np.asarray(scale, float) + np.asarray(offset, float)
    mg.compute_metrics(m)
    x = (m.C - m.C.mean(0)) / np.asarray(scale, float)
    _compare(m, [np.random.default_rng(1).random(m.n_cells), np.clip(0.5 - x @ [3.0, 2.0, 1.0], 0, 1)])
