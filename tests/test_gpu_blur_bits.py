"""The sparse blur's blocks of pixels make the bits of its definition: tap by tap in the reference's order, each operation
rounded to the output's type (fused for float and double)."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def by_definition(image, k, sigma):
    """Every pixel convolved (torchhull gaussian_blur_cuda.cu:205-286), the x offset outside.  A float tap is fused: its
    product is exact in 64 bits, where the sum is rounded before it is rounded to 32, which differs from rounding once only
    where 29 further bits are a one and zeros, or a zero and ones.  A double tap is exact where image values are 0 or 1."""
    r, (h, w) = k // 2, image.shape[1:]
    dtype = image.dtype
    offsets = torch.arange(-r, r + 1, device=image.device)
    square = (offsets[:, None] ** 2 + offsets[None, :] ** 2).float()
    weights = torch.exp(-square / torch.tensor(2.0 * sigma * sigma, dtype=torch.float32, device=image.device)).to(dtype)
    ys = [reflected(d, h, image.device) for d in range(-r, r + 1)]
    xs = [reflected(d, w, image.device) for d in range(-r, r + 1)]
    total = torch.zeros((), dtype=dtype, device=image.device)
    acc = torch.zeros_like(image)
    for i in range(k):
        for j in range(k):
            weight, value = weights[i, j], image[:, ys[j]][:, :, xs[i]]
            total = total + weight
            if dtype == torch.float16:
                acc = acc + weight * value
            else:
                acc = (acc.double() + weight.double() * value.double()).to(dtype)
    return (acc.float() / total.float()).half() if dtype == torch.float16 else acc / total


def reflected(d, n, device):
    """image_utils.h:129-160; a position of exactly -(n - 1) is taken for 0 there."""
    if n == 1:
        return torch.zeros(n, dtype=torch.int64, device=device)
    at, m = torch.arange(n, device=device) + d, n - 1
    flips = torch.div(at, m, rounding_mode="trunc") + (at < 0)
    return torch.where(flips % 2 == 0, at % m, m - at % m)


def active(image, k):
    """Pixels of the k/2 x k/2 tiles that hold an edge pixel, and of the tiles around those."""
    r, (h, w) = k // 2, image.shape[1:]
    edge = torch.zeros(image.shape, dtype=torch.bool, device=image.device)
    edge[:, :, :-1] |= image[:, :, :-1] != image[:, :, 1:]
    edge[:, :-1] |= image[:, :-1] != image[:, 1:]
    tiles = torch.nn.functional.pad(edge[:, None].float(), (0, (w // r + 1) * r - w, 0, (h // r + 1) * r - h))
    tiles = torch.nn.functional.max_pool2d(torch.nn.functional.max_pool2d(tiles, r), 3, stride=1, padding=1)[:, 0]
    return tiles.repeat_interleave(r, 1).repeat_interleave(r, 2)[:, :h, :w] > 0


# one block of 32 x 32 pixels, its edges, sizes that are no multiples of it, and one smaller than the kernel's reach
@pytest.mark.parametrize("size", [(32, 32), (33, 31), (70, 101), (5, 40), (129, 64)])
@pytest.mark.parametrize("k", [3, 5, 7, 9, 11, 13, 17, 25])
@pytest.mark.parametrize("dtype,soft", [(torch.float16, False), (torch.float16, True), (torch.float32, False), (torch.float32, True),
                                        (torch.float64, False)])
def test_same_bits(th, cuda, dtype, soft, k, size):
    g = torch.Generator().manual_seed(1000 * k + size[0])
    image = torch.rand((2, *size), generator=g)
    image[:, :, size[1] // 2 :] = (image[:, :, size[1] // 2 :] < 0.03).float()  # few edges: pixels that are left alone
    image = (image if soft else (image < 0.5).float()).to(dtype).to(cuda)
    got = th.gaussian_blur(image[..., None].contiguous(), k, 2.0)[..., 0]
    want = torch.where(active(image, k), by_definition(image, k, 2.0), image)
    assert torch.equal(got, want)
