"""The plane solve with a warp per cell (short lists) and with filled warps, on
both sides of the line between them, against the serial CPU oracle, bit for
bit: list lengths that leave warps and groups part-filled, all cell classes,
cells whose bisection meets coinciding levels or alpha itself."""

import numpy as np
import pytest

from geometricvofext_gb300 import capi, meshgen as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("kind,n", [("hex", 13), ("jitter", 13), ("tet", 8), ("checker", 11), ("refined", 12)])
def test_both_sides_of_the_line(kind, n, split):
    import torch

    line = 8 * torch.cuda.get_device_properties(0).multi_processor_count
    m = mg.make_mesh(kind, n)
    assert m.n_cells > line + 7
    g = capi.Simplic(m, split_warped_face=split)
    o = O.Oracle(m, split_warped_face=bool(split))
    rng = np.random.default_rng(11)
    for k in (2, line - 1, line, line + 1, line + 7):
        pick = rng.choice(m.n_cells, k, replace=False)
        for name, v in (("random", rng.random(k)), ("halves", rng.choice([0.5, 0.25, 1e-7, 1 - 1e-7], k))):
            a = (rng.random(m.n_cells) < 0.5).astype(float)
            a[pick] = v
            g.reconstruct(a)
            o.reconstruct(a)
            for x, y, what in zip(g.mixed(), o.mixed(), ("cells", "statuses")):
                np.testing.assert_array_equal(x, y, err_msg=f"{k} {name}: {what}")
            assert len(g.mixed()[0]) == k
            for x, y, what in zip(g.interface(), o.interface(), "NDCS"):
                np.testing.assert_array_equal(x, y, err_msg=f"{k} {name}: interface{what}")
