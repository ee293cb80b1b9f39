"""The blur's blocks of 32 x 32 pixels at their edges: sizes around blocks, wide kernels, rows that vector loads cannot take."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu

# images (batch, height, width): below, at and above one or two blocks of 32 x 32 pixels; smaller than the halo; odd rows
SHAPES = [(2, 31, 63), (1, 32, 64), (3, 33, 65), (1, 70, 130), (1, 5, 7)]


def images(shape, dtype, seed):
    rng = np.random.default_rng(seed)
    m = np.zeros((*shape, 1))
    for b in range(shape[0]):
        y, x = int(rng.integers(shape[1])), int(rng.integers(shape[2]))
        m[b, : y + 1, : x + 1] = 1.0  # a corner of ones: most tiles hold no edge
    if dtype.is_floating_point:
        m *= rng.uniform(0.25, 1.0)
    return torch.from_numpy(m).to(dtype)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kernel_size", [3, 5, 15, 17, 33, 75])
@pytest.mark.parametrize("sparse", [True, False])
@pytest.mark.parametrize("in_dtype,out_dtype", [(torch.float32, torch.float32), (torch.uint8, torch.float32),
                                                (torch.float64, torch.float64), (torch.int64, torch.float64)])
def test_blocks_match_oracle(th, cuda, shape, kernel_size, sparse, in_dtype, out_dtype):
    m = images(shape, in_dtype, 100 * kernel_size + shape[2])
    got = th.gaussian_blur(m.to(cuda), kernel_size, 2.0, sparse, out_dtype).cpu().double().numpy()
    ref = oracle.gaussian_blur(m, kernel_size, 2.0, sparse, dtype=str(out_dtype).split(".")[1]).astype(np.float64)
    # values of at most 1, weights that add up to 1: k^2 additions of relative error 2^-24 each on either side,
    # and weights (float32 expf of host and device) and their sum a few 2^-23 off
    tol = 2 * (kernel_size**2 + 8) * 2.0**-24 if out_dtype == torch.float32 else 16 * 2.0**-23
    assert np.abs(got - ref).max() <= tol


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kernel_size", [3, 9])
@pytest.mark.parametrize("sparse", [True, False])
def test_half_blocks_match_oracle(th, cuda, shape, kernel_size, sparse):
    m = images(shape, torch.float16, 7 + shape[1])
    got = th.gaussian_blur(m.to(cuda), kernel_size, 2.0, sparse).cpu().float().numpy()
    ref = oracle.gaussian_blur(m, kernel_size, 2.0, sparse, dtype="float16").astype(np.float32)
    assert np.abs(got - ref).max() <= 3e-3  # as for the other half results


@pytest.mark.parametrize("dtype", [torch.uint8, torch.float16, torch.float32])
def test_vector_and_scalar_rows_agree(th, cuda, dtype):
    """The same pixels, once in rows of a 16-byte multiple and once shifted off that alignment."""
    m = images((2, 40, 80), dtype, 3).to(cuda)
    out_dtype = torch.float32 if dtype == torch.uint8 else dtype
    off = torch.empty(m.numel() + 1, dtype=dtype, device=cuda)[1:].view(m.shape)
    off.copy_(m)
    assert torch.equal(th.gaussian_blur(m, 9, 2.0, True, out_dtype), th.gaussian_blur(off, 9, 2.0, True, out_dtype))


def test_special_values_pass_through(th, cuda):
    """Infinities and NaN spread over their kernel's reach only, and flat infinite regions are copied."""
    m = torch.zeros(1, 96, 192, 1)
    m[0, 40, 100] = float("nan")
    m[0, :20, :40] = float("inf")
    got = th.gaussian_blur(m.to(cuda), 5, 1.0, True).cpu()[0, ..., 0]
    assert torch.isnan(got[38:43, 98:103]).all() and not torch.isnan(got[34:47, 106:]).any()
    assert torch.isinf(got[:10, :30]).all() and (got[60:] == 0).all()
