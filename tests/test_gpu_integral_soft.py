"""Integral images of masks between 0 and 1: heights around the rows a thread has in flight, widths and row counts around a 32x32 tile."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("height,width", [(1, 1), (31, 32), (32, 31), (33, 64), (63, 65), (64, 33), (65, 1), (97, 96), (1, 300), (129, 130)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32, torch.float64])
def test_same_additions_in_the_same_order(th, cuda, height, width, dtype):
    g = torch.Generator().manual_seed(height * 11 + width)
    m = torch.rand((3, height, width, 1), generator=g).to(dtype)
    # one sequential float32 sum down each column, then one along each row: every bit is fixed
    ref = np.cumsum(np.cumsum(m[..., 0].float().numpy(), axis=1, dtype=np.float32), axis=2, dtype=np.float32)
    out = th.integral_image(m.to(cuda)).reshape(3, height, width).cpu().numpy()
    assert np.array_equal(out.view(np.int32), ref.view(np.int32))
