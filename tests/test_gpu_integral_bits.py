"""Integral images of 0/1 masks from bit words: heights around a band of 32 rows and around the bands a block counts itself."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def exact(masks):
    return torch.cumsum(torch.cumsum(masks[..., 0].double(), 1), 2).float()


@pytest.mark.parametrize("height,width", [(1, 1), (31, 33), (32, 128), (33, 130), (64, 4), (1024, 36), (1025, 37), (1056, 260),
                                          (40, 8192), (40, 8196), (5, 100001)])
@pytest.mark.parametrize("dtype", [torch.uint8, torch.float16, torch.float32, torch.float64])
def test_bands(th, cuda, height, width, dtype):
    g = torch.Generator().manual_seed(height * 7 + width)
    m = (torch.rand((2, height, width, 1), generator=g) < 0.6).to(dtype).to(cuda)
    assert torch.equal(th.integral_image(m).reshape(2, height, width), exact(m))


def test_all_ones_up_to_the_largest_exact_sum(th, cuda):
    m = torch.ones((1, 4096, 4096, 1), device=cuda)
    out = th.integral_image(m).reshape(4096, 4096)
    assert out[-1, -1].item() == 2**24 and torch.equal(out, exact(m)[0])


def test_one_other_value_in_the_last_band(th, cuda):
    m = torch.ones((2, 65, 40, 1), device=cuda)
    m[1, 64, 39] = 0.25
    out = th.integral_image(m).reshape(2, 65, 40)
    ref = torch.cumsum(torch.cumsum(m[..., 0], 1), 2)
    assert torch.equal(out, ref)
