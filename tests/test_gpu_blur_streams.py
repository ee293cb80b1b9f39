"""Blurs of one context on several streams share its scratch: each gets its own result."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sparse", [True, False])
def test_interleaved_streams(th, cuda, sparse):
    g = torch.Generator().manual_seed(17)
    images = [(torch.rand((8, 300 + 40 * i, 500, 1), generator=g) < 0.5).float().to(cuda) for i in range(4)]
    want = [th.gaussian_blur(m, 9, 2.0, sparse=sparse) for m in images]
    streams = [torch.cuda.Stream() for _ in images]
    torch.cuda.synchronize()
    got = [[] for _ in images]
    for _ in range(8):
        for i, (m, s) in enumerate(zip(images, streams)):
            with torch.cuda.stream(s):
                got[i].append(th.gaussian_blur(m, 9, 2.0, sparse=sparse))
    torch.cuda.synchronize()
    for i, w in enumerate(want):
        assert all(torch.equal(w, o) for o in got[i])


@pytest.mark.parametrize("sparse", [True, False])
def test_interleaved_weights(th, cuda, sparse):
    """Images of one shape: every call writes its own weights to the same place."""
    g = torch.Generator().manual_seed(18)
    image = (torch.rand((8, 400, 500, 1), generator=g) < 0.5).float().to(cuda)
    sigmas = [0.7, 1.5, 2.5, 4.0]
    want = [th.gaussian_blur(image, 9, s, sparse=sparse) for s in sigmas]
    streams = [torch.cuda.Stream() for _ in sigmas]
    torch.cuda.synchronize()
    got = [[] for _ in sigmas]
    for _ in range(8):
        for i, (sigma, s) in enumerate(zip(sigmas, streams)):
            with torch.cuda.stream(s):
                got[i].append(th.gaussian_blur(image, 9, sigma, sparse=sparse))
    torch.cuda.synchronize()
    for i, w in enumerate(want):
        assert all(torch.equal(w, o) for o in got[i])
