"""Plane solve of refined box cells (faces and edges split by their smaller
neighbours), whose vertex levels are settled in single precision, against the
CPU oracle bit for bit: any proportions, size and place, nearly axis-aligned
planes, cells that no longer fill their bounding box."""

import numpy as np
import pytest

from geometricvofext_gb300 import capi, meshgen as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n", [("checker", 8), ("refined", 8)])
@pytest.mark.parametrize("scale,offset,shear", [((1, 1, 1), (0, 0, 0), 0), ((1, 0.01, 30), (-5, 0.3, 2), 0),
                                                ((1e-4, 1e-4, 1e-4), (0, 0, 0), 0), ((1e-7, 1, 1), (0, 0, 0), 0),
                                                ((1, 1, 1), (3e7, 0, 0), 0), ((1, 1, 1), (0, 0, 0), 1e-3),
                                                ((1, 1, 1), (0, 0, 0), 1e-7)])
def test_refined_boxes_bitexact(kind, n, scale, offset, shear):
    m = mg.make_mesh(kind, n)
    m.points = m.points * np.asarray(scale, float) + np.asarray(offset, float)
    m.points[:, 0] += shear * m.points[:, 1]
    mg.compute_metrics_general(m)
    rng = np.random.default_rng(5)
    g, o = capi.Simplic(m), O.Oracle(m)
    x = (m.C - m.C.mean(0)) / np.asarray(scale, float)
    for name, a in (("random", rng.random(m.n_cells)), ("steep", rng.random(m.n_cells) ** 12),
                    ("plane", np.clip(0.5 - x @ [3.0, 2.0, 1.0], 0, 1)), ("slab", np.clip(0.5 - 4 * x[:, 1], 0, 1)),
                    ("tilted slab", np.clip(0.5 - x @ [1e-4, 4.0, 1e-7], 0, 1))):
        g.reconstruct(a)
        o.reconstruct(a)
        for p, q, what in zip(g.mixed(), o.mixed(), ("cells", "statuses")):
            np.testing.assert_array_equal(p, q, err_msg=f"{name}: {what}")
        for p, q, what in zip(g.interface(), o.interface(), "NDCS"):
            np.testing.assert_array_equal(p, q, err_msg=f"{name}: interface{what}")
