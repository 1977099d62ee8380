"""Plane solve against the CPU oracle, bit for bit, where the given cell
volumes are not those of the cells' geometry: the bisection over the vertex
levels compares cut volume / V with alpha."""

import numpy as np
import pytest

from geometricvofext_gb300 import capi, meshgen as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n", [("hex", 6), ("hex", 12), ("checker", 6)])
@pytest.mark.parametrize("spread", [1e-9, 1e-5, 1e-3, 0.3])
def test_given_volumes_decide_the_levels(kind, n, spread):
    m = mg.make_mesh(kind, n)
    rng = np.random.default_rng(n)
    m.V = m.V * (1.0 + spread * rng.uniform(-1, 1, m.n_cells))
    g, o = capi.Simplic(m), O.Oracle(m)
    for name, a in (("random", rng.random(m.n_cells)), ("one in eight", np.where(rng.random(m.n_cells) < 0.125, 0.6, 0.0))):
        g.reconstruct(a)
        o.reconstruct(a)
        for p, q, what in zip(g.mixed(), o.mixed(), ("cells", "statuses")):
            np.testing.assert_array_equal(p, q, err_msg=f"{name}: {what}")
        for p, q, what in zip(g.interface(), o.interface(), "NDCS"):
            np.testing.assert_array_equal(p, q, err_msg=f"{name}: interface{what}")
