"""The mixed form's normals and interface speeds by several lanes per cell and
by one thread per cell: a cell whose surroundings are the same gets the same
bits whatever the length of the list it is in (the line between the two lies
between the lists compared here)."""

import numpy as np
import pytest

from geometricvofext_gb300 import capi, harness as H, meshgen as mg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n", [("hex", 37), ("jitter", 37), ("tet", 21)])
def test_same_bits_in_short_and_long_lists(kind, n):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    m = mg.make_mesh(kind, n)
    assert 300 * sms < m.n_cells and m.n_cells < 2 * 240 * sms
    g = capi.Simplic(m, precision=capi.PRECISION_MIXED, n_alpha_bounds=0, clip=0)
    flow = H.DeformationFlow(m)
    dt = H.cfl_delta_t(m, flow.phi0)
    a = np.random.default_rng(9).uniform(0.01, 0.99, m.n_cells)
    x = m.C[:, 0]
    half = np.where(x < 0.5, a, 0.0)
    few = np.where(x < 0.2, a, 0.0)
    out = []
    for f in (a, half, few):
        g.reconstruct(f)
        count, N = len(g.mixed()[0]), g.interface()[0]
        g.advect(f, flow.phi0, flow.U0, dt, U_boundary=flow.Ub)
        out.append((count, N, g.alpha_phi()))
    assert out[0][0] == m.n_cells and out[1][0] < 240 * sms
    xf = m.Cf[:, 0]
    for k, lim in ((1, 0.5), (2, 0.2)):
        inner = np.flatnonzero(x < lim - 3.0 / n)  # all of the stencil alike
        np.testing.assert_array_equal(out[k][1][inner], out[0][1][inner])
        faces = np.flatnonzero(xf < lim - 3.0 / n)
        np.testing.assert_array_equal(out[k][2][faces], out[0][2][faces])
