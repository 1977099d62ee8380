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


@pytest.mark.parametrize("scale,offset", [((1, 1, 1), (0, 0, 0)), ((1, 0.01, 30), (-5, 0.3, 2)),
                                          ((1e-4, 1e-4, 1e-4), (0, 0, 0)), ((1e-7, 1, 1), (0, 0, 0)),
                                          ((1, 1, 1), (3e7, 0, 0)), ((2e-3, 3e-3, 1e-3), (1e4, -1e4, 0))])
def test_box_shortcuts_bitexact(scale, offset):
    """Box cells of any proportions, size and place: the axis-aligned faces'
    short forms and the single precision level test keep the oracle's bits,
    also where they have to give way to the full operations."""
    m = mg.hex_mesh(6, metrics=False)
    m.points = m.points * np.asarray(scale, float) + np.asarray(offset, float)
    mg.compute_metrics(m)
    rng = np.random.default_rng(5)
    g, o = capi.Simplic(m), O.Oracle(m)
    x = (m.C - m.C.mean(0)) / np.asarray(scale, float)
    for name, a in (("random", rng.random(m.n_cells)), ("steep", rng.random(m.n_cells) ** 12),
                    ("plane", np.clip(0.5 - x @ [3.0, 2.0, 1.0], 0, 1)), ("slab", np.clip(0.5 - 4 * x[:, 1], 0, 1)),
                    ("tilted slab", np.clip(0.5 - x @ [1e-4, 4.0, 1e-7], 0, 1))):
        g.reconstruct(a)
        o.reconstruct(a)
        for p, q, what in zip(g.interface(), o.interface(), "NDCS"):
            np.testing.assert_array_equal(p, q, err_msg=f"{name}: interface{what}")
