"""The item kernel's last level, whose items a block shares: few views and cells, and blocks whose last warps have no parent."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle
from torchhull_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("views,level", [(1, 4), (2, 5), (5, 7), (13, 6), (40, 5)])
@pytest.mark.parametrize("partial", [False, True])
def test_last_level(th, cuda, views, level, partial):
    r = scenes.make_request(900 + views, views, 128, level, partial, n_capsules=4 if partial else 0, device=cuda)
    th._C.set_carve_kernel(0, 2)
    try:
        got = th.visual_hull(**r.kwargs())
    finally:
        th._C.set_carve_kernel(0, 0)
    ref = oracle.visual_hull(r.masks.cpu(), r.transforms.cpu(), r.level, r.cube_corner_bfl, r.cube_length, r.masks_partial,
                             r.transforms_convention, r.unique_verts)
    assert np.array_equal(got[0].cpu().numpy(), ref.verts) and np.array_equal(got[1].cpu().numpy(), ref.faces)
