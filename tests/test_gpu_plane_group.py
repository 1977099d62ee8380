"""The group plane solve (a group of lanes per cell) against the serial CPU
oracle, bit for bit, on fields where every cell is mixed: 1 to a few hundred
cells (part-filled warps and groups, all cell classes), random normals,
planes along faces and diagonals (levels that coincide, sub-faces of no area)
and volume fractions at the ends of the mixed range."""

import numpy as np
import pytest

from geometricvofext_gb300 import capi, meshgen as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _fields(m, rng):
    n, C = m.n_cells, m.C
    yield "random", rng.random(n)
    yield "one cell", np.where(np.arange(n) == n // 2, 0.37, 0.0)
    yield "slab", np.clip(0.5 - (C[:, 2] - 0.43) * 3, 0, 1)
    yield "slab with noise", np.clip(0.5 - (C[:, 2] - 0.43) * 3 + 1e-9 * rng.standard_normal(n), 0, 1)
    yield "diagonal", np.clip(0.5 - (C.sum(1) - 1.3) * 2, 0, 1)
    yield "ends", rng.choice([2e-8, 1e-6, 0.3, 1 - 1e-7, 1.0, 0.0, 1 - 3e-8], n)


@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("kind,n", [("hex", 3), ("hex", 7), ("jitter", 6), ("tet", 4), ("checker", 6), ("refined", 8)])
def test_planes_bitexact_on_rough_fields(kind, n, split):
    m = mg.make_mesh(kind, n)
    g = capi.Simplic(m, split_warped_face=split)
    o = O.Oracle(m, split_warped_face=bool(split))
    for name, a in _fields(m, np.random.default_rng(3)):
        g.reconstruct(a)
        o.reconstruct(a)
        for x, y, what in zip(g.mixed(), o.mixed(), ("cells", "statuses")):
            np.testing.assert_array_equal(x, y, err_msg=f"{name}: {what}")
        for x, y, what in zip(g.interface(), o.interface(), "NDCS"):
            np.testing.assert_array_equal(x, y, err_msg=f"{name}: interface{what}")
