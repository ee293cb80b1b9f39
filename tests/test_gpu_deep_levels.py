"""Hulls of levels 11 and 12: rows of more than 32 words of 64 points, row flags counted ahead, no cell masks."""

from __future__ import annotations

import functools

import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu

CORNER, LENGTH = (-1.0, -1.0, -1.0), 2.0


def rod(side, width, tilt):
    """Two views of a rod `width` pixels of 2 / side across that runs along x through the whole cube; view 1 looks along z,
    view 2 along y."""
    masks = torch.zeros((2, side, 16, 1))
    masks[:, (side - width) // 2 : (side + width) // 2] = 1.0
    transforms = torch.zeros((2, 4, 4))
    transforms[:, 0, 0] = 0.5
    transforms[0, 1, 1] = transforms[1, 1, 2] = 1.0
    transforms[:, 1, 0] = tilt
    transforms[:, 3, 3] = 1.0
    return masks, transforms


@functools.cache
def expected(level, unique):
    # a pixel is as wide as two cells at level 11, as four at level 12
    masks, transforms = rod(1024, 6 if level == 11 else 3, 0.013)
    return oracle.visual_hull(masks, transforms, level, CORNER, LENGTH, False, "opengl", unique)


@pytest.mark.parametrize("unique", [True, False])
@pytest.mark.parametrize("level", [11, 12])
def test_mesh(th, cuda, level, unique):
    masks, transforms = rod(1024, 6 if level == 11 else 3, 0.013)
    verts, faces = th.visual_hull(masks.to(cuda), transforms.to(cuda), level, CORNER, LENGTH, False, "opengl", unique)
    want = expected(level, unique)
    assert len(want.faces) > 0
    assert np.array_equal(verts.cpu().numpy(), want.verts) and np.array_equal(faces.cpu().numpy(), want.faces)


@pytest.mark.parametrize("level", [11, 12])
def test_field(th, cuda, level):
    masks, transforms = rod(1024, 6 if level == 11 else 3, 0.013)
    index, values, r = th._C.sparse_visual_hull_field_raw(masks.to(cuda), transforms.to(cuda), level, CORNER, LENGTH, False, "opengl")
    want = expected(level, True)
    assert r == (1 << level) + 1
    assert (want.field_indices % r).max() == r - 1  # the last word of a row
    assert np.array_equal(index.cpu().numpy(), want.field_indices) and np.array_equal(values.cpu().numpy(), want.field_values)
