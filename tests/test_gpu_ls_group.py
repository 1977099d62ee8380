"""Least-squares normals and the isoRDF orientation by 16 lanes per cell and by
one thread per cell, on both sides of the lines between them, against the CPU
oracle bit for bit: stencils of 8 to some 100 cells, singular fits, lists that
leave half a warp idle."""

import numpy as np
import pytest

from geometricvofext_gb300 import capi, meshgen as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _same(g, o, a):
    g.reconstruct(a)
    o.reconstruct(a)
    for x, y, what in zip(g.mixed(), o.mixed(), ("cells", "statuses")):
        np.testing.assert_array_equal(x, y, err_msg=what)
    for x, y, what in zip(g.interface(), o.interface(), "NDCS"):
        np.testing.assert_array_equal(x, y, err_msg=f"interface{what}")


@pytest.mark.parametrize("kind,n", [("hex", 2), ("hex", 19), ("jitter", 19), ("tet", 11), ("checker", 8), ("refined", 8)])
def test_normals(kind, n):
    import torch

    line = 40 * torch.cuda.get_device_properties(0).multi_processor_count
    m = mg.make_mesh(kind, n)
    g, o = capi.Simplic(m), O.Oracle(m)
    rng = np.random.default_rng(4)
    _same(g, o, rng.random(m.n_cells))
    _same(g, o, np.full(m.n_cells, 0.5))  # no gradient
    for k in (1, line, line + 1):
        if k > m.n_cells:
            continue
        a = np.zeros(m.n_cells)
        a[rng.choice(m.n_cells, k, replace=False)] = rng.uniform(1e-3, 0.999, k)
        _same(g, o, a)


@pytest.mark.parametrize("kind,n", [("hex", 19), ("hex", 30), ("jitter", 10), ("tet", 6), ("checker", 8), ("refined", 8)])
def test_iso_rdf(kind, n):
    m = mg.make_mesh(kind, n)
    g, o = capi.Simplic(m, orientation_method=capi.ORIENTATION_ISO_RDF), O.Oracle(m, orientation="isoRDF")
    x = m.C
    _same(g, o, np.random.default_rng(5).random(m.n_cells))
    _same(g, o, np.clip(0.5 + n * (0.3 - np.linalg.norm(x - 0.47, axis=1)), 0, 1))
