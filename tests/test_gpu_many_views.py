"""More than 32 views: the second word of the carve's view masks, views beyond both words, and the batch that mixes them."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle
from torchhull_gb300 import scenes

pytestmark = pytest.mark.gpu


def reference(r):
    return oracle.visual_hull(r.masks.cpu(), r.transforms.cpu(), r.level, r.cube_corner_bfl, r.cube_length, r.masks_partial,
                              r.transforms_convention, r.unique_verts)


def same(got, ref):
    return np.array_equal(got[0].cpu().numpy(), ref.verts) and np.array_equal(got[1].cpu().numpy(), ref.faces)


@pytest.mark.parametrize("views", [31, 32, 33, 63, 64, 65, 70])
@pytest.mark.parametrize("partial,convention", [(False, "opengl"), (True, "opencv")])
@pytest.mark.parametrize("kernel", [1, 2])
def test_views_around_a_mask_word(th, cuda, views, partial, convention, kernel):
    r = scenes.make_request(700 + views, views, 96, 6, partial, convention, n_capsules=4 if partial else 0, device=cuda)
    th._C.set_carve_kernel(0, kernel)
    try:
        got = th.visual_hull(**r.kwargs())
    finally:
        th._C.set_carve_kernel(0, 0)
    assert same(got, reference(r))


def test_batch_mixes_mask_words(th, cuda):
    reqs = [scenes.make_request(800 + v, v, 96, level, partial, n_capsules=4 if partial else 0, device=cuda)
            for v, level, partial in ((8, 6, False), (48, 6, True), (70, 5, False), (33, 6, False))]
    outs = th._C.visual_hull_batch([(r.masks, r.transforms, r.level, r.cube_corner_bfl, r.cube_length, r.masks_partial,
                                     r.transforms_convention, r.unique_verts) for r in reqs])
    for got, r in zip(outs, reqs):
        assert same(got, reference(r))
