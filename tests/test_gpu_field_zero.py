"""The sparse field's values are those of a coalesced tensor: sums from 0, so never -0."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("views", [3, 4])
def test_no_negative_zero(th, cuda, views):
    """Negative masks whose corners project outside every image: a zero sample per view, and an odd
    number of negative ones among the factors make the product -0."""
    masks = torch.full((views, 2, 2, 1), -0.5, device=cuda)
    transforms = torch.zeros((views, 4, 4), device=cuda)
    transforms[:, 2, 3] = transforms[:, 3, 3] = 1.0
    transforms[:, 0, 3] = transforms[:, 1, 3] = 1.0  # OpenCV: every point falls on the pixel position (0.5, 0.5)
    transforms[-1, 0, 3] = 100.0  # the last view: outside the image
    args = (masks, transforms, 0, (0.0, 0.0, 0.0), 1.0, False, "opencv")
    raw = th._C.sparse_visual_hull_field_raw(*args)[1]
    assert raw.numel() == 8 and (raw == 0).all() and torch.signbit(raw).all() == (views % 2 == 0)
    field = th.sparse_visual_hull_field(*args)
    want = torch.sparse_coo_tensor(field.indices(), raw, field.shape).coalesce()
    assert field.is_coalesced() and torch.equal(field.indices(), want.indices())
    assert torch.equal(field.values().view(torch.int32), want.values().view(torch.int32))
